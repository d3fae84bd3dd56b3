"""Parity of the CUDA embedding path with the CPU oracle and with the reference's
known-answer tests, through the C ABI.  Bit-exact for ids, rows, COO indices and
for sums over sorted segment ids; 1e-5 relative for the atomic (unsorted) route."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from oracle import oracle
from tests.golden import reference_cases as rc

pytestmark = pytest.mark.gpu

import torch
from annc_b200 import ops  # noqa: E402  (no fallback: a missing library fails the collection)
from annc_b200 import AnncError, synth  # noqa: E402
from annc_b200._lib import ALLOC_FN, lib  # noqa: E402
from annc_b200.device import BagPlan  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("case", rc.SEGMENT_REDUCE, ids=lambda c: c["name"])
@pytest.mark.parametrize("where", ["host", "device"])
def test_segment_reduce_golden(case, where):
    args = [case["data"], case["indices"], case["slice_input"]]
    if where == "device":
        args = [_dev(a) for a in args]
    out, so = ops.kp_fused_sparse_segment_reduce(*args, case["begin"], case["begin_1"], case["combiner"])
    if where == "device":
        out, so = out.cpu().numpy(), so.cpu().numpy()
    np.testing.assert_array_equal(out, case["out"])
    assert int(so) == case["slice_out"]


@pytest.mark.parametrize("mut", rc.SEGMENT_REDUCE_ERRORS, ids=lambda m: m[2][:24])
def test_segment_reduce_errors(mut):
    base = dict(rc.SEGMENT_REDUCE[1])
    base[mut[0]] = mut[1]
    with pytest.raises(AnncError) as e:
        ops.kp_fused_sparse_segment_reduce(base["data"], base["indices"], base["slice_input"],
                                           base["begin"], base["begin_1"], 0)
    assert mut[2] in e.value.message


@pytest.mark.parametrize("dim", [1, 3, 4, 8, 12, 16, 32, 64, 100, 128, 130, 256, 512])
@pytest.mark.parametrize("combiner", [0, 1])
@pytest.mark.parametrize("idx_dtype", [np.int32, np.int64])
def test_segment_reduce_sorted_bit_exact(dim, combiner, idx_dtype):
    rng = np.random.default_rng(dim * 7 + combiner)
    rows, batch = 997, 301
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    lens = rng.integers(0, 7, batch)  # empty bags included
    lens[-1] = max(lens[-1], 1)
    nnz = int(lens.sum())
    seg = np.repeat(np.arange(batch), lens)
    slice_input = np.stack([rng.integers(0, 9, nnz), seg, rng.integers(0, 9, nnz)], 1).astype(np.int64)
    idx = rng.integers(0, rows, nnz).astype(idx_dtype)
    begin, begin_1 = np.array([0, 1], np.int32), np.array([0], np.int32)
    want, want_so = oracle.sparse_segment_reduce(data, idx, slice_input, begin, begin_1, combiner)
    got, so = ops.kp_fused_sparse_segment_reduce(_dev(data), _dev(idx), _dev(slice_input), begin, begin_1, combiner)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert int(so.cpu()) == int(want_so)


@pytest.mark.parametrize("combiner", [0, 1])
def test_segment_reduce_unsorted(combiner):
    rng = np.random.default_rng(5)
    rows, batch, dim, nnz = 500, 64, 64, 3000
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    seg = rng.integers(0, batch, nnz)
    slice_input = np.stack([seg, np.zeros(nnz, np.int64)], 1).astype(np.int64)
    idx = rng.integers(0, rows, nnz).astype(np.int64)
    begin, begin_1 = np.array([0, 0], np.int32), np.array([1], np.int32)
    want, want_so = oracle.sparse_segment_reduce(data, idx, slice_input, begin, begin_1, combiner)
    got, so = ops.kp_fused_sparse_segment_reduce(data, idx, slice_input, begin, begin_1, combiner)
    scale = np.abs(want).max()
    assert np.abs(got - want).max() <= 1e-5 * scale  # fp32 pooling tolerance, order not fixed
    assert int(so) == int(want_so)


def test_segment_reduce_empty_and_single():
    data = np.arange(12, dtype=np.float32).reshape(3, 4)
    begin, b1 = np.array([0, 0], np.int32), np.array([0], np.int32)
    out, so = ops.kp_fused_sparse_segment_reduce(data, np.zeros(0, np.int32), np.zeros((0, 2), np.int64), begin, b1, 0)
    np.testing.assert_array_equal(out, np.zeros((1, 4), np.float32))  # max starts at 0 -> batch 1
    assert int(so) == 1
    out, _ = ops.kp_fused_sparse_segment_reduce(data, np.array([2], np.int32), np.array([[5, 0]], np.int64), begin, b1, 1)
    want = np.zeros((6, 4), np.float32)
    want[5] = data[2]
    np.testing.assert_array_equal(out, want)


def test_segment_reduce_row_out_of_range_is_reported():
    data = np.ones((4, 8), np.float32)
    with pytest.raises(AnncError):
        ops.kp_fused_sparse_segment_reduce(data, np.array([0, 9], np.int32), np.array([[0, 0], [1, 0]], np.int64),
                                           np.array([0, 0], np.int32), np.array([0], np.int32), 0)


@pytest.mark.parametrize("case", rc.SEGMENT_REDUCE_NONZERO, ids=lambda c: c["name"])
def test_segment_reduce_nonzero_golden(case):
    shp, idx, val = ops.kp_fused_sparse_segment_reduce_nonzero(
        case["data"], case["indices"], case["slice_input"], case["begin"], case["combiner"])
    np.testing.assert_array_equal(shp, case["out_shape"])
    np.testing.assert_array_equal(idx, case["out_indices"])
    np.testing.assert_array_equal(val, case["out_values"])


@pytest.mark.parametrize("mut", rc.SEGMENT_REDUCE_NONZERO_ERRORS, ids=lambda m: m[2][:24])
def test_segment_reduce_nonzero_errors(mut):
    base = dict(rc.SEGMENT_REDUCE_NONZERO[1])
    base[mut[0]] = mut[1]
    with pytest.raises(AnncError) as e:
        ops.kp_fused_sparse_segment_reduce_nonzero(base["data"], base["indices"], base["slice_input"], base["begin"], 0)
    assert mut[2] in e.value.message


@pytest.mark.parametrize("rank,combiner", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_segment_reduce_nonzero_random(rank, combiner):
    rng = np.random.default_rng(rank * 2 + combiner)
    rows, dim, nnz = 211, 12, 5000
    data = rng.integers(-2, 3, (rows, dim)).astype(np.float32)  # many exact zeros in the sums
    if rank == 1:
        data = data[:, 0].copy()
    seg = np.sort(rng.integers(0, 400, nnz))
    seg = seg + 1000  # sparse, large segment ids: first-appearance ranks differ from ids
    slice_input = np.stack([np.zeros(nnz, np.int64), seg], 1).astype(np.int64)
    idx = rng.integers(0, rows, nnz).astype(np.int32)
    begin = np.array([0, 1], np.int32)
    w_shp, w_idx, w_val = oracle.sparse_segment_reduce_nonzero(data, idx, slice_input, begin, combiner)
    shp, gi, gv = ops.kp_fused_sparse_segment_reduce_nonzero(_dev(data), _dev(idx), _dev(slice_input), begin, combiner)
    np.testing.assert_array_equal(shp.cpu().numpy(), w_shp)
    np.testing.assert_array_equal(gi.cpu().numpy(), w_idx)
    np.testing.assert_array_equal(gv.cpu().numpy(), w_val)


@pytest.mark.parametrize("case", rc.FUSED_GATHER, ids=lambda c: c["name"])
def test_fused_gather_golden(case):
    u, inv, rows = ops.kp_fused_gather(case["data"], case["keys"], case["begin"])
    np.testing.assert_array_equal(u, case["unique"])
    np.testing.assert_array_equal(inv, case["indices"])
    np.testing.assert_array_equal(rows, case["out"])


@pytest.mark.parametrize("err", rc.FUSED_GATHER_ERRORS, ids=lambda e: e[3][:20])
def test_fused_gather_errors(err):
    data, keys, begin, msg = err
    with pytest.raises(AnncError) as e:
        ops.kp_fused_gather(data, keys, begin)
    assert msg in e.value.message


def test_fused_gather_random_first_appearance():
    rng = np.random.default_rng(11)
    rows, dim, nnz = 5000, 24, 40000
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    keys = np.stack([rng.integers(0, 7, nnz), rng.zipf(1.3, nnz) % rows], 1).astype(np.int64)
    begin = np.array([0, 1], np.int32)
    wu, wi, wr = oracle.fused_gather(data, keys, begin)
    u, inv, r = ops.kp_fused_gather(_dev(data), _dev(keys), begin)
    np.testing.assert_array_equal(u.cpu().numpy(), wu)
    np.testing.assert_array_equal(inv.cpu().numpy(), wi)
    np.testing.assert_array_equal(r.cpu().numpy(), wr)


@pytest.mark.parametrize("case", rc.DYNAMIC_STITCH, ids=lambda c: c["name"])
def test_dynamic_stitch_golden(case):
    np.testing.assert_array_equal(ops.kp_fused_sparse_dynamic_stitch(case["x"], case["tables"]), case["out"])


@pytest.mark.parametrize("err", rc.DYNAMIC_STITCH_ERRORS, ids=lambda e: e[2][:20])
def test_dynamic_stitch_errors(err):
    x, tables, msg = err
    with pytest.raises(AnncError) as e:
        ops.kp_fused_sparse_dynamic_stitch(x, tables)
    assert msg in e.value.message


def test_dynamic_stitch_random():
    rng = np.random.default_rng(3)
    n_part, dim = 5, 64
    tabs = [rng.standard_normal((int(r), dim)).astype(np.float32) for r in rng.integers(100, 400, n_part)]
    limit = min(t.shape[0] for t in tabs) * n_part
    x = rng.integers(0, limit, (37, 41)).astype(np.int64)
    want = oracle.sparse_dynamic_stitch(x, tabs)
    got = ops.kp_fused_sparse_dynamic_stitch(_dev(x), [_dev(t) for t in tabs])
    np.testing.assert_array_equal(got.cpu().numpy(), want)


EDGE_IDS = np.array([0, 1, 999_999, 1_000_000, 1_000_001, (1 << 62) - 1, (1 << 63) - 1, (1 << 63),
                     (1 << 64) - 1, 0x9E3779B97F4A7C15], np.uint64)


@pytest.mark.parametrize("num_buckets", [1, 2, 7, 1000, 1_000_000])
@pytest.mark.parametrize("bounded", [False, True])
def test_hash_bucket_gather_bit_exact(num_buckets, bounded):
    rng = np.random.default_rng(num_buckets)
    rows = num_buckets if not bounded else max(1, num_buckets // 2)
    rows = min(rows, 50_000)
    nb = num_buckets if bounded else rows
    w = rng.standard_normal((rows, 64)).astype(np.float32)
    fp = np.concatenate([EDGE_IDS, rng.integers(0, 1 << 63, 5000, dtype=np.uint64) * np.uint64(2) + np.uint64(1)])
    empty = rng.random(fp.shape[0]) < 0.1
    want = oracle.embedding_with_hash_bucket(fp, empty, w, nb, bounded=bounded)
    got = ops.kp_fused_embedding_with_hash_bucket(_dev(fp.view(np.int64)).view(torch.int64), _dev(w), nb,
                                                  empty=_dev(empty), bounded=bounded)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    got_h = ops.kp_fused_embedding_with_hash_bucket(fp, w, nb, empty=empty, bounded=bounded)
    np.testing.assert_array_equal(got_h, want)


def test_sparse_embedding_matches_reference_quirk():
    rng = np.random.default_rng(9)
    fp = rng.integers(0, 1 << 63, 300, dtype=np.uint64)
    fp[::7] = np.uint64(50) * fp[::7]  # multiples of num_buckets -> bucket 0 -> value dropped
    empty = rng.random(300) < 0.2
    wi, wv, we, ws = oracle.sparse_embedding(fp, empty, 50)
    gi, gv, ge, gs = ops.kp_fused_sparse_embedding(fp, 50, empty=empty)
    np.testing.assert_array_equal(gi, wi)
    np.testing.assert_array_equal(gv, wv)
    np.testing.assert_array_equal(ge, we)
    np.testing.assert_array_equal(gs, ws)
    assert len(gv) < len(gi)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_sparse_embedding2(dtype):
    rng = np.random.default_rng(2)
    table = rng.standard_normal((100, 16)).astype(np.float32)
    ids = rng.integers(-20, 140, 1000).astype(dtype)
    want = oracle.sparse_embedding2(ids, table, 0, 100, 0)
    got = ops.sparse_embedding2(_dev(ids), _dev(table), 0, 100, 0)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    np.testing.assert_array_equal(ops.sparse_embedding2(ids, table, 0, 100, 0), want)


@pytest.mark.parametrize("combiner", [0, 1])
def test_grouped_hash_bags_bit_exact(combiner):
    """embed_hash_bucket + segment pooling for several tables in one launch, output
    interleaved as [batch, slots, dim] the way the DLRM pipeline consumes it."""
    rows = [1000, 37, 250_000, 5]
    w = synth.embedding_workload(4, rows, 64, 2048, 20, 1.05)
    slots = len(rows) + 1
    out = torch.full((2048, slots, 64), 7.0, device="cuda")
    plan = BagPlan([_dev(t) for t in w.tables], [_dev(b.raw_ids) for b in w.bags],
                   [_dev(b.slice_input) for b in w.bags], out, 1, 2048, id_kind=2, col=0, combiner=combiner)
    plan.run()
    assert plan.error_bits() == 0
    got = out.cpu().numpy()
    assert (got[:, 0, :] == 7.0).all()  # slot 0 untouched
    for t, (tab, bag) in enumerate(zip(w.tables, w.bags)):
        idx = oracle.hash_bucket(bag.raw_ids.view(np.uint64), rows[t])
        want, _ = oracle.sparse_segment_reduce(tab, idx, bag.slice_input, np.array([0, 0], np.int32),
                                               np.array([0], np.int32), combiner)
        np.testing.assert_array_equal(got[:, t + 1, :], want)


def test_hash_bags_full_size_properties():
    """Config-sized run (26 tables x 1M x 64, batch 16384) checked through properties that
    need no full CPU pass: linearity in the table values and an exact check on a slice."""
    w = synth.hash_bucket_bag_case(seed=0, tables=26, rows=1_000_000, batch=16384)
    tabs = [_dev(t) for t in w.tables]
    ids = [_dev(b.raw_ids) for b in w.bags]
    segs = [_dev(b.slice_input) for b in w.bags]
    out = torch.empty((16384, 26, 64), device="cuda")
    plan = BagPlan(tabs, ids, segs, out, 0, 16384, id_kind=2, col=0, combiner=0)
    plan.run()
    assert plan.error_bits() == 0
    base = out.clone()
    for t in (0, 13, 25):
        idx = oracle.hash_bucket(w.bags[t].raw_ids.view(np.uint64), 1_000_000)
        want, _ = oracle.sparse_segment_reduce(w.tables[t], idx, w.bags[t].slice_input,
                                               np.array([0, 0], np.int32), np.array([0], np.int32), 0)
        np.testing.assert_array_equal(base[:, t, :].cpu().numpy(), want)
    # scaling every table by 2 (exact in fp32) must scale every pooled vector by 2
    for t in tabs:
        t.mul_(2.0)
    plan.run()
    assert torch.equal(out, base * 2.0)


@pytest.mark.parametrize("shards,combiner", [(2, 0), (3, 1), (8, 0)])
def test_row_sharded_exchange_on_one_gpu(shards, combiner):
    """The fused pooling + exchange step with its ranks run one after the other on one GPU:
    each rank pools the lookups it owns (mod partition) into its part of a receive buffer and
    leaves bags it does not contribute to unwritten (the buffer is poisoned with NaN first);
    the owner mask, computed from the ids alone, must name exactly the written parts, and the
    masked rank-order sum must match the unsharded oracle within the fp32 pooling tolerance."""
    from annc_b200.device import BagLaunch, BagPrepass, OwnerMask, sum_partials_masked
    rows = [1000, 37, 50_000, 5, 3]
    B, D = 1024, 64
    T = len(rows)
    w = synth.embedding_workload(11, rows, D, B, 12, 1.05)
    dev = torch.device("cuda")
    ids = [_dev(b.raw_ids) for b in w.bags]
    segs = [_dev(b.slice_input) for b in w.bags]
    pre = BagPrepass(segs, B)
    ws = torch.zeros(pre.ws_bytes, dtype=torch.uint8, device=dev)
    pre.run(ws)
    off_ptr = lambda t: ws.data_ptr() + 512 + t * (B + 1) * 4
    recv = torch.full((shards, B, T, D), float("nan"), device=dev)
    keep = []
    for g in range(shards):
        shard_tabs = [_dev(np.ascontiguousarray(t[g::shards]) if t[g::shards].shape[0] else
                           np.zeros((1, D), np.float32)) for t in w.tables]
        keep.append(shard_tabs)
        entries = [(shard_tabs[t].data_ptr(), len(range(g, rows[t], shards)), rows[t],
                    ids[t].data_ptr(), None, ids[t].shape[0],
                    recv.data_ptr() + ((g * B) * T + t) * D * 4, off_ptr(t)) for t in range(T)]
        launch = BagLaunch(entries, D, B, 2, T * D, dev, combiner=combiner, shard_count=shards,
                           shard_rank=g, exchange=True)
        launch.run()
        assert launch.error_bits() == 0
    owners = OwnerMask([(ids[t].data_ptr(), ids[t].shape[0], rows[t], off_ptr(t)) for t in range(T)],
                       B, shards, dev)
    owners.run()
    mask = owners.mask.cpu().numpy().reshape(T, B)
    written = ~torch.isnan(recv[:, :, :, 0]).cpu().numpy()  # [shards, B, T]
    for t, bag in enumerate(w.bags):
        bucket = bag.raw_ids.view(np.uint64) % np.uint64(rows[t])
        want_mask = np.zeros(B, np.int64)
        np.bitwise_or.at(want_mask, bag.slice_input[:, 0], 1 << (bucket % np.uint64(shards)).astype(np.int64))
        np.testing.assert_array_equal(mask[t], want_mask)
        for g in range(shards):
            np.testing.assert_array_equal(written[g, :, t], (want_mask >> g) & 1 == 1)
    out = torch.full((B, T, D), 3.0, device=dev)
    sum_partials_masked(recv.data_ptr(), owners.mask, shards, B * T * D, B, T, D, out.data_ptr(), T * D)
    got = out.cpu().numpy()
    for t, (tab, bag) in enumerate(zip(w.tables, w.bags)):
        idx = oracle.hash_bucket(bag.raw_ids.view(np.uint64), rows[t])
        want, _ = oracle.sparse_segment_reduce(tab, idx, bag.slice_input, np.array([0, 0], np.int32),
                                               np.array([0], np.int32), combiner)
        scale = max(float(np.abs(want).max()), 1e-30)
        assert float(np.abs(got[:, t, :] - want).max()) / scale <= 1e-5


@pytest.mark.parametrize("num_buckets", [1, 2, 3, 7, 10**6, 2**31 - 1, 2**32 + 1, 2**62 + 3, 2**63 - 1])
def test_division_free_modulo_is_exact(num_buckets):
    """The kernels compute `fingerprint % num_buckets` with a reciprocal multiply and a
    correction step.  The owner-mask kernel exposes (id % num_buckets) % G without needing a
    table of num_buckets rows; three coprime G pin the bucket on edge and random ids."""
    from annc_b200.device import OwnerMask
    rng = np.random.default_rng(3)
    d = num_buckets
    edge = [0, 1, d - 1, d, d + 1, 2 * d - 1, 2 * d, 2**62 - 1, 2**63 - 1, 2**63, 2**64 - 1,
            2**64 - d, (2**64 - 1) // d * d, (2**64 - 1) // d * d - 1]
    ids = np.array([e % 2**64 for e in edge if e >= 0], dtype=np.uint64)
    ids = np.concatenate([ids, rng.integers(0, 2**64, 4096, dtype=np.uint64)])
    n = ids.shape[0]
    ids_d = _dev(ids.view(np.int64))
    off = _dev(np.arange(n + 1, dtype=np.int32))  # one lookup per bag
    want_bucket = np.array([int(x) % d for x in ids.tolist()], dtype=object)
    for g in (32, 31, 29):
        m = OwnerMask([(ids_d.data_ptr(), n, d, off.data_ptr())], n, g, torch.device("cuda"))
        m.run()
        got = m.mask.cpu().numpy().view(np.uint32)
        want = np.array([1 << (int(b) % g) for b in want_bucket], dtype=np.uint32)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dim,stride_slots", [(4, 1), (20, 2), (48, 3), (64, 3), (128, 2), (132, 1), (256, 2), (264, 1), (516, 1)])
@pytest.mark.parametrize("combiner", [0, 1])
@pytest.mark.parametrize("id_kind", [0, 1, 2])
def test_bag_plan_tile_and_chunk_edges(dim, stride_slots, combiner, id_kind):
    """Grouped bags at the lengths where the lookup-granular kernel can go wrong: lookups around a
    tile and a chunk, one bag over many chunks, runs of empty bags at either end and in between, a
    table without lookups, widths that fill the lanes of a row only partly.  Bit-exact: both sides
    add a bag's rows in lookup order."""
    rng = np.random.default_rng(dim + 10 * combiner + id_kind)
    rows, batch = 211, 1300
    cases = [np.bincount([5], minlength=batch), np.bincount([batch - 1] * 7, minlength=batch),
             np.bincount([0] * 8 + [1299], minlength=batch), np.bincount([700] * 2000, minlength=batch),
             np.zeros(batch, np.int64), rng.integers(0, 3, batch) * rng.integers(0, 9, batch),
             np.full(batch, 1), np.where(np.arange(batch) % 100 == 50, 31, 0), np.full(batch, 17)]
    tabs, ids, segs, want = [], [], [], []
    for lens in cases:
        n = int(lens.sum())
        data = rng.standard_normal((rows, dim)).astype(np.float32)
        raw = rng.integers(0, 1 << 62, n) if id_kind == 2 else rng.integers(0, rows, n)
        row = raw % rows
        seg = np.stack([np.repeat(np.arange(batch), lens), rng.integers(0, 9, n)], 1).astype(np.int64)
        ref = np.zeros((batch, dim), np.float32)
        np.add.at(ref, seg[:, 0], data[row])
        if combiner:
            ref *= (np.float32(1) / np.maximum(lens, 1).astype(np.float32))[:, None]
        tabs.append(_dev(data))
        ids.append(_dev(raw.astype(np.int32 if id_kind == 0 else np.int64)))
        segs.append(_dev(seg.reshape(n, 2)))
        want.append(ref)
    slots = len(cases) + stride_slots
    out = torch.full((batch, slots, dim), -7.0, device="cuda")
    plan = BagPlan(tabs, ids, segs, out, stride_slots, batch, id_kind=id_kind, combiner=combiner)
    plan.run()
    got = out.cpu().numpy()
    assert plan.error_bits() == 0
    assert (got[:, :stride_slots] == -7.0).all()
    for t, ref in enumerate(want):
        np.testing.assert_array_equal(got[:, stride_slots + t], ref, err_msg=f"table {t}")


@pytest.mark.parametrize("dim", [64, 252, 256, 260])
@pytest.mark.parametrize("combiner", [0, 1])
def test_bag_plan_marks_unsorted_and_out_of_range(dim, combiner):
    """A table whose segment ids decrease is redone by the atomic route (sums in any order: as many ulp
    of the sum of magnitudes as a bag has lookups), its neighbours are not; a row or segment id out of
    range is reported and added nowhere."""
    rng = np.random.default_rng(dim + combiner)
    rows, batch, n = 300, 200, 3000
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    row, lens = rng.integers(0, rows, n), rng.multinomial(n, np.ones(batch) / batch)
    seg = np.repeat(np.arange(batch), lens)
    shuffled = rng.permutation(seg)
    out = torch.full((batch, 3, dim), -7.0, device="cuda")
    pairs = [np.stack([s, s], 1).astype(np.int64) for s in (seg, shuffled, seg)]
    plan = BagPlan([_dev(data)] * 3, [_dev(row)] * 3, [_dev(p) for p in pairs], out, 0, batch, id_kind=1, combiner=combiner)
    plan.run()
    assert plan.error_bits() == 0
    got = out.cpu().numpy()
    for t, s in enumerate((seg, shuffled, seg)):
        ref, size = np.zeros((batch, dim)), np.zeros((batch, dim))
        np.add.at(ref, s, data[row].astype(np.float64))
        np.add.at(size, s, np.abs(data[row]).astype(np.float64))
        div = np.maximum(np.bincount(s, minlength=batch), 1)[:, None] if combiner else 1
        assert (np.abs(got[:, t] - ref / div) <= (lens.max() + 2) * 2.0 ** -24 * size / div + 1e-30).all()
    assert np.array_equal(got[:, 0], got[:, 2])
    bad_row, bad_seg = row.copy(), pairs[0].copy()
    bad_row[17], bad_seg[n - 1] = rows, batch
    for ids, sg, bit in ((bad_row, pairs[0], 1), (row, bad_seg, 2)):
        plan = BagPlan([_dev(data)], [_dev(ids)], [_dev(sg)], out, 1, batch, id_kind=1, combiner=0)
        plan.run()
        assert plan.error_bits() == bit


@pytest.mark.parametrize("dim", [4, 8, 40, 64, 72, 256, 512])
@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("combiner", [0, 1])
def test_bags_around_the_decoded_window(dim, shift, combiner):
    """Bags that end anywhere in the short windows of a call of few lookups (chunks of 16 or 24, then windows of 128) and
    reach over several, tables 32-byte aligned and not, rows out of range among them: the sums in lookup
    order, bit for bit."""
    rng = np.random.default_rng(dim + shift)
    rows, lens = 300, []
    for n in (1, 223, 1, 31, 32, 33, 224, 225, 255, 256, 257, 700, 127, 128, 129, 0, 0, 3, 1500, 1):
        lens += [n] + list(rng.integers(0, 4, 5))
    lens = np.array(lens * 12)
    batch, n = len(lens), int(lens.sum())
    seg = np.repeat(np.arange(batch), lens)
    idx = rng.integers(0, rows, n)
    idx[rng.integers(0, n, 5)] = rows + 3
    base = torch.zeros(rows * dim + 4, device="cuda")
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    table = base[shift:shift + rows * dim].view(rows, dim)
    table.copy_(_dev(data))
    out = torch.empty((batch, 1, dim), device="cuda")
    plan = BagPlan([table], [_dev(idx)], [_dev(np.stack([seg, seg], 1).astype(np.int64))], out, 0, batch, id_kind=1,
                   combiner=combiner)
    plan.run()
    want = np.zeros((batch, dim), np.float32)
    ok = idx < rows
    np.add.at(want, seg[ok], data[idx[ok]])  # in order, in fp32
    if combiner:
        want *= (np.float32(1) / np.maximum(lens, 1).astype(np.float32))[:, None]
    assert plan.error_bits() == 1
    np.testing.assert_array_equal(out.cpu().numpy()[:, 0], want)


def _hash_bags(rng, lens):
    """Raw ids and index matrix of one table's bags."""
    seg = np.repeat(np.arange(len(lens)), lens)
    ids = rng.integers(0, 1 << 62, len(seg))
    return ids, np.stack([seg, seg], 1).astype(np.int64).reshape(-1, 2)


def _oracle_bags(tables, ids, segs, batch, combiner):
    want = np.full((batch, len(tables), tables[0].shape[1]), np.nan, np.float32)
    oracle.embed_bags_tables(tables, [t.shape[0] for t in tables], ids, segs, batch, tables[0].shape[1], want, len(tables),
                             0, combiner=combiner, threads=oracle.host_threads())
    return want


@pytest.mark.parametrize("dim", [12, 32, 40, 64, 100, 128, 160, 256, 512])
@pytest.mark.parametrize("shift,id_kind", [(0, 2), (4, 1), (0, 0)])
@pytest.mark.parametrize("bags", ["long", "short"])
def test_bags_around_a_full_window(dim, shift, id_kind, bags):
    """Enough lookups for the longest chunks (4736 resident warps of 224, 3552 above 256 floats): bags that end at, just
    before and just behind the chunk, the 32 lookups behind it and the windows of 128 after that, in rows that
    are 32-byte aligned and not, by four and by eight rows a round, every kind of id: the oracle's sums, bit for bit."""
    rng = np.random.default_rng(dim + shift)
    n_all = (3552 if dim > 256 else 4736) * 224
    edges = [224] * 6 + [223, 1, 225, 31, 193, 32, 192, 33, 191, 255, 256, 257, 383, 384, 385, 512, 0, 0, 1500, 127, 128, 129]
    lens = []
    while sum(lens) < n_all // 8:  # an eighth of the lookups in bags that the edges are about
        lens += edges + list(rng.integers(0, 5, rng.integers(0, 30)))
    hi = 60 if bags == "long" else 9
    fill = rng.integers(0, hi, 2 * (n_all - sum(lens)) // (hi - 1))
    at = np.sort(rng.integers(0, len(fill), 40))
    lens = np.concatenate([v for part in zip(np.array_split(np.array(lens), 41), np.split(fill, at)) for v in part])
    batch, rows = len(lens), 3000
    ids, pairs = _hash_bags(rng, lens)
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    base = torch.zeros(rows * dim + 4, device="cuda")
    table = base[shift:shift + rows * dim].view(rows, dim)
    table.copy_(_dev(data))
    out = torch.full((batch, 1, dim), np.nan, device="cuda")
    given = ids if id_kind == 2 else ids.astype(np.uint64) % rows
    plan = BagPlan([table], [_dev(given.astype(np.int32 if id_kind == 0 else np.int64))], [_dev(pairs)], out, 0, batch,
                   id_kind=id_kind, combiner=id_kind == 1)
    plan.run()
    assert plan.error_bits() == 0
    np.testing.assert_array_equal(out.cpu().numpy(), _oracle_bags([data], [ids], [pairs], batch, int(id_kind == 1)))


@pytest.mark.parametrize("dim", [8, 16, 36, 64, 100, 128, 256, 512])
@pytest.mark.parametrize("batch", [300, 12000])
@pytest.mark.parametrize("share", [0, 3])
def test_tables_of_different_bag_lengths(dim, batch, share):
    """Tables of one call with bags of one, of a few, of many lookups, with very long ones among short ones and with none
    at all: chunks of a length per table, the oracle's sums bit for bit; with a share of the SMs too."""
    rng = np.random.default_rng(dim * batch)
    u = lambda lo, hi: rng.integers(lo, hi + 1, batch)
    lens = [np.ones(batch, int), u(20, 80), u(0, 1), np.zeros(batch, int), u(1, 3), np.where(u(0, 99) == 0, 400, 1), u(1, 20),
            np.where(np.arange(batch) == batch - 1, 1, 0)]
    ids, segs = zip(*(_hash_bags(rng, v) for v in lens))
    tables = [rng.standard_normal((int(r), dim)).astype(np.float32) for r in rng.integers(1, 2000, len(lens))]
    out = torch.full((batch, len(lens), dim), np.nan, device="cuda")
    lib.annc_embed_bag_set_stream_ctas_per_sm(share)
    try:
        plan = BagPlan([_dev(t) for t in tables], [_dev(i) for i in ids], [_dev(s) for s in segs], out, 0, batch)
        plan.run()
        assert plan.error_bits() == 0
    finally:
        lib.annc_embed_bag_set_stream_ctas_per_sm(0)
    np.testing.assert_array_equal(out.cpu().numpy(), _oracle_bags(tables, ids, segs, batch, 0))


@pytest.mark.parametrize("dim", [16, 32, 64, 100, 128])
def test_bag_share_fits_beside_the_pooling_kernel(dim):
    """A share of n blocks per SM leaves room for 5 - n blocks of the pooling kernel of the row exchange
    (256 threads of at most 48 registers, by its launch bounds), and gives the same sums."""
    rng = np.random.default_rng(dim)
    rows, batch = 500, 3000
    lens = rng.integers(0, 12, batch)
    n = int(lens.sum())
    seg = np.repeat(np.arange(batch), lens)
    out = torch.empty((batch, 1, dim), device="cuda")
    plan = BagPlan([_dev(rng.standard_normal((rows, dim)).astype(np.float32))], [_dev(rng.integers(0, rows, n))],
                   [_dev(np.stack([seg, seg], 1).astype(np.int64))], out, 0, batch, id_kind=1, combiner=1)
    plan.run()
    want = out.clone()
    try:
        for share in (1, 2, 3, 4, 5):
            lib.annc_embed_bag_set_stream_ctas_per_sm(share)
            regs = C.c_int(0)
            assert lib.annc_embed_bag_stream_registers(dim, C.byref(regs)) == 0
            resident = min(share, 65536 // (256 * regs.value))
            assert 256 * (resident * regs.value + (5 - share) * 48) <= 65536, (share, regs.value)
            out.fill_(-7.0)
            plan.run()
            assert plan.error_bits() == 0 and torch.equal(out, want)
    finally:
        lib.annc_embed_bag_set_stream_ctas_per_sm(0)


@pytest.mark.parametrize("n,distinct,dim", [(1, 1, 4), (2047, 3, 5), (2048, 2048, 8), (2049, 700, 20), (10_000, 1, 64),
                                            (70_001, 30_000, 16), (4_300_000, 9_000, 1)])
def test_gather_unique_tiles(n, distinct, dim):
    """Unique keys in first-appearance order at the edges of the counting tiles, with one key that
    holds most positions, and beyond the size where the tiles are summed in a pass of their own."""
    rng = np.random.default_rng(n)
    rows = distinct + 5
    pool = rng.permutation(rows)[:distinct]
    keys = np.where(rng.random(n) < 0.5, pool[0], pool[rng.integers(0, distinct, n)])
    keys[rng.permutation(n)[:min(n, distinct)]] = pool[:min(n, distinct)]
    data = rng.standard_normal((rows, dim)).astype(np.float32)
    col = np.stack([np.arange(n), keys], 1).astype(np.int64)
    uniq, inv, got = ops.kp_fused_gather(_dev(data), _dev(col), np.array([0, 1], np.int32))
    u, first, idx = np.unique(keys, return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")
    rank = np.empty(len(u), np.int64)
    rank[order] = np.arange(len(u))
    np.testing.assert_array_equal(uniq.cpu().numpy(), u[order])
    np.testing.assert_array_equal(inv.cpu().numpy(), rank[idx])
    np.testing.assert_array_equal(got.cpu().numpy(), data[u[order]])


@pytest.mark.parametrize("bad", [-1, 50])
def test_gather_and_reduce_report_rows_outside_the_table(bad):
    data = _dev(np.ones((50, 8), np.float32))
    keys = np.stack([np.zeros(300, np.int64), np.arange(300) % 50], 1)
    keys[299, 1] = bad
    with pytest.raises(AnncError) as e:
        ops.kp_fused_gather(data, _dev(keys), np.array([0, 1], np.int32))
    assert "idx out of table range" in e.value.message
    with pytest.raises(AnncError) as e:
        ops.kp_fused_sparse_segment_reduce(data, _dev(keys[:, 1].copy()), _dev(np.sort(keys.clip(0), axis=0)),
                                           np.zeros(2, np.int32), np.zeros(1, np.int32), 0)
    assert "indices out of range" in e.value.message


@pytest.mark.parametrize("nnz", [0, 1, 511, 512, 4095, 4096, 4097, 9000])
@pytest.mark.parametrize("shuffled", [False, True])
def test_segment_reduce_at_the_edges_of_the_scan(nnz, shuffled):
    """The scan for the output's size by one block and by several; its flags reach the host (unsorted ids,
    rows out of range), call after call from the same thread."""
    rng = np.random.default_rng(nnz)
    data = rng.standard_normal((70, 8)).astype(np.float32)
    seg = np.sort(rng.integers(0, nnz // 3 + 1, nnz))
    if shuffled:
        seg = rng.permutation(seg)
    idx = rng.integers(0, 70, nnz)
    pairs = np.stack([seg, seg], 1).astype(np.int64).reshape(nnz, 2)
    b2, b1 = np.zeros(2, np.int32), np.zeros(1, np.int32)
    for _ in range(3):
        out, so = ops.kp_fused_sparse_segment_reduce(_dev(data), _dev(idx), _dev(pairs), b2, b1, 0)
    batch = int(seg.max()) + 1 if nnz else 1
    want = np.zeros((batch, 8), np.float32)
    np.add.at(want, seg, data[idx])
    assert int(so) == batch and tuple(out.shape) == (batch, 8)
    if shuffled:  # sums of up to a few dozen rows in any order
        np.testing.assert_allclose(out.cpu().numpy(), want, rtol=0, atol=1e-5)
    else:
        np.testing.assert_array_equal(out.cpu().numpy(), want)
    if nnz:
        idx[nnz - 1] = 70
        with pytest.raises(AnncError):
            ops.kp_fused_sparse_segment_reduce(_dev(data), _dev(idx), _dev(pairs), b2, b1, 0)


def test_one_operator_call_per_thread():
    """Threads one after the other, each with a single call that waits for a posted size: a thread must not take
    what was posted for one that has ended, whose pinned memory it may be given, for its own."""
    rng = np.random.default_rng(5)
    data = rng.standard_normal((50, 8)).astype(np.float32)
    d_data, zeros = _dev(data), (np.zeros(2, np.int32), np.zeros(1, np.int32))
    good = []

    def call(i):
        n = [9000, 40, 5000, 700][i // 2 % 4] + i
        seg, idx = rng.integers(0, n // (2 + i // 4), n), rng.integers(0, 50, n)
        if i % 3:
            seg = np.sort(seg)
        pairs = _dev(np.stack([idx, seg], 1).astype(np.int64))
        if i % 2:
            unique, inverse, rows = (o.cpu().numpy() for o in ops.kp_fused_gather(d_data, pairs, zeros[0]))
            want = idx[np.sort(np.unique(idx, return_index=True)[1])]
            assert np.array_equal(unique, want) and np.array_equal(want[inverse], idx)
            assert np.array_equal(rows, data[want])
        else:
            out, so = ops.kp_fused_sparse_segment_reduce(d_data, _dev(idx), pairs, np.array([0, 1], np.int32), zeros[1], 0)
            want, size = np.zeros((2, seg.max() + 1, 8)), np.bincount(seg)[:, None]
            np.add.at(want[0], seg, data[idx])
            np.add.at(want[1], seg, np.abs(data[idx]))
            assert int(so) == len(size) == out.shape[0]
            assert (np.abs(out.cpu().numpy() - want[0]) <= 2.0 ** -24 * size * want[1]).all()  # adds in any order
        good.append(i)

    for i in range(32):
        t = threading.Thread(target=call, args=(i,))
        t.start()
        t.join()
    assert good == list(range(32))


@pytest.mark.parametrize("refused", [0, 1, 2])
@pytest.mark.parametrize("begin_on_device", [False, True])
def test_calls_that_fail_between_their_kernels_leave_none_running(refused, begin_on_device):
    """An output allocation that fails after the size was posted: the kernels behind the one that posted it write the
    caller's other outputs, so the stream is idle when the call returns, and the next call is not disturbed."""
    rng = np.random.default_rng(refused)
    n, dim = 2_000_000, 8
    data = _dev(rng.standard_normal((300_000, dim)).astype(np.float32))
    key = rng.integers(0, 300_000, n)
    keys, idx = _dev(np.stack([key, np.sort(key)], 1)), _dev(key)
    begin = np.array([0, 1], np.int32)
    want = [o.cpu().numpy() for o in ops.kp_fused_gather(data, keys, begin)]
    total = ops.kp_fused_sparse_segment_reduce(data, idx, keys, begin, begin[:1], 0)[0].cpu().numpy()
    if begin_on_device:
        begin = _dev(begin)
    outs = ops._outputs_for(data)

    @ALLOC_FN
    def alloc(ctx, index, dtype, rank, dims):
        return None if index == refused else outs._alloc(ctx, index, dtype, rank, dims)

    t, b = ops.as_tensor, C.byref
    first = begin[:1]
    for _ in range(5):
        rc = lib.annc_KPFusedGather(b(t(data)), b(t(keys)), b(t(begin)), alloc, None)
        assert rc != 0 and torch.cuda.current_stream().query()
        if refused < 2:
            rc = lib.annc_KPFusedSparseSegmentReduce(b(t(data)), b(t(idx)), b(t(keys)), b(t(begin)), b(t(first)), C.c_int(0),
                                                     alloc, None)
            assert rc != 0 and torch.cuda.current_stream().query()
    for got, w in zip(ops.kp_fused_gather(data, keys, begin), want):
        np.testing.assert_array_equal(got.cpu().numpy(), w)
    np.testing.assert_array_equal(ops.kp_fused_sparse_segment_reduce(data, idx, keys, begin, first, 0)[0].cpu().numpy(), total)


_BLOCKING = """
import ctypes, time
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0 and cuda.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0  # CU_CTX_SCHED_BLOCKING_SYNC
import numpy as np, torch
from annc_b200 import ops
data, begin = torch.randn((1000, 8), device="cuda"), np.array([0, 1], np.int32)
key = torch.arange(20000, device="cuda") % 700
keys = torch.stack([key, key.sort()[0]], 1)
x = torch.randn((8192, 8192), device="cuda")
calls = [lambda: ops.kp_fused_gather(data, keys, begin),
         lambda: ops.kp_fused_sparse_segment_reduce(data, key, keys, begin, begin[:1], 0)]
for call in calls:
    call(), torch.mm(x, x)
    torch.cuda.synchronize()
    for _ in range(10):
        torch.mm(x, x)
    wall, busy = time.perf_counter(), time.thread_time()
    call()
    wall, busy = time.perf_counter() - wall, time.thread_time() - busy
    assert wall > 0.05 and busy < wall / 4, (wall, busy)  # tens of GFLOP of fp32 ahead: the thread sleeps
"""


def test_posted_results_are_waited_for_as_the_application_asked():
    """With the device set to blocking waits, a call behind a long queue leaves its core to others."""
    r = subprocess.run([sys.executable, "-c", _BLOCKING], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


@pytest.mark.parametrize("where", ["host", "device"])
def test_an_operator_inside_the_allocation_of_another(monkeypatch, where):
    """An operator that runs while another's output is allocated (an allocator's hook, a finalizer) leaves the outer
    call its outputs."""
    put = _dev if where == "device" else np.asarray
    data = put(np.arange(40, dtype=np.float32).reshape(10, 4))
    keys = put(np.array([[0, 3], [1, 7], [2, 3]], np.int64))
    begin, inner, outer = np.array([0, 1], np.int32), [], []
    plain = ops._Outputs._alloc

    def alloc(self, ctx, index, dtype, rank, dims):
        outer[:] = outer or [self]
        if self is outer[0]:  # before each of its three outputs, in the middle of its scratch
            inner.append(ops.kp_fused_gather(data, put(np.array([[0, 9], [1, 8], [2, 9]], np.int64)), begin))
        return plain(self, ctx, index, dtype, rank, dims)

    monkeypatch.setattr(ops._Outputs, "_alloc", alloc)
    calls = [ops.kp_fused_gather(data, keys, begin)] + inner
    assert len(calls) == 4
    for (unique, inverse, rows), want in zip(calls, ([3, 7], [9, 8], [9, 8], [9, 8])):
        assert unique.tolist() == want and inverse.tolist() == [0, 1, 0] and rows.tolist() == data[want].tolist()


@pytest.mark.parametrize("n", [50, 5000, 400_000])
def test_gather_and_reduce_behind_the_kernels_that_make_their_operands(n):
    """Keys, segment ids and rows written by kernels that are still running when the operators are called, call after call
    over the same buffers."""
    g = torch.Generator(device="cuda").manual_seed(n)
    heavy = torch.randn((4096, 4096), device="cuda", generator=g)
    rows, zeros = 1000, np.zeros(2, np.int32)
    data, pairs = torch.zeros((rows, 16), device="cuda"), torch.zeros((n, 2), dtype=torch.int64, device="cuda")
    sources = [(torch.randn((rows, 16), device="cuda", generator=g),
                torch.stack([torch.randint(0, hi, (n,), device="cuda", generator=g),
                             torch.sort(torch.randint(0, n // hi + 1, (n,), device="cuda", generator=g))[0]], 1))
               for hi in (7, rows, 300, 1)]

    def calls(wait):
        out = []
        for d, p in sources:
            torch.mm(heavy, heavy)
            data.copy_(d)
            pairs.copy_(p)
            wait()
            out += list(ops.kp_fused_gather(data, pairs, zeros))
            out.append(ops.kp_fused_sparse_segment_reduce(data, pairs[:, 0].contiguous(), pairs, np.array([0, 1], np.int32),
                                                          zeros[:1], 0)[0])
        return out

    want = calls(torch.cuda.synchronize)
    for _ in range(3):
        for a, b in zip(calls(lambda: None), want):
            assert torch.equal(a, b)
