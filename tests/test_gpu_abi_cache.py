"""The host-pointer side of the ABI: device mirrors of host operands keyed by (pointer, bytes),
uploads skipped when the sampled fingerprint of the host contents is unchanged (weights upload
once; an output that comes back as the next call's input is not uploaded), the re-laid kn4
weight kept with its mirror, and the report of a tensor-core wait that ran out.  The staging
counters of the library (annc_staging_counters) are the evidence."""
import ctypes as C

import numpy as np
import pytest
import torch

from annc_b200 import ops
from annc_b200._lib import lib
from oracle import oracle

pytestmark = pytest.mark.gpu


def counters():
    a, b, c = C.c_uint64(0), C.c_uint64(0), C.c_uint64(0)
    lib.annc_staging_counters(C.byref(a), C.byref(b), C.byref(c))
    return a.value, b.value, c.value


def nerr(got, want):
    return float(np.abs(got - want).max() / max(np.abs(want).max(), 1e-30))


@pytest.fixture(autouse=True)
def _default_mode():
    lib.annc_set_operand_cache(2, 0)
    yield
    lib.annc_set_operand_cache(2, 0)


def test_second_call_with_the_same_weight_uploads_nothing():
    rng = np.random.default_rng(0)
    m, k, n = 256, 384, 512
    x = rng.standard_normal((m, k)).astype(np.float32)
    w = rng.standard_normal((k, n)).astype(np.float32)
    addend = np.ascontiguousarray(np.broadcast_to(rng.standard_normal(n).astype(np.float32), (m, n)))
    zeros = np.zeros((m, n), np.float32)
    out = np.empty((m, n), np.float32)
    info = [ops.shape_info(addend), ops.shape_info(addend), ops.shape_info(x), ops.shape_info(w)]
    operands = [zeros, addend, x, w] + info
    want = oracle.matmul_add_relu(addend, x, w)

    h0, d0, s0 = counters()
    ops._call_custom("__matmul_add_relu", out, operands)
    h1, d1, s1 = counters()
    assert h1 - h0 == x.nbytes + w.nbytes + addend.nbytes  # the max operand is never read
    assert d1 - d0 == out.nbytes
    assert nerr(out, want) <= 2e-3

    out[:] = -1
    ops._call_custom("__matmul_add_relu", out, operands)
    h2, d2, s2 = counters()
    assert h2 - h1 == 0, "weight, addend and activation are unchanged: nothing to upload"
    assert s2 - s1 == x.nbytes + w.nbytes + addend.nbytes
    assert nerr(out, want) <= 2e-3

    # a new batch in the same buffer: only the activation travels
    x[:] = rng.standard_normal((m, k)).astype(np.float32)
    ops._call_custom("__matmul_add_relu", out, operands)
    h3, _, _ = counters()
    assert h3 - h2 == x.nbytes
    assert nerr(out, oracle.matmul_add_relu(addend, x, w)) <= 2e-3

    # mode 1: constants (weight, addend) are reused, activations always travel
    lib.annc_set_operand_cache(1, 0)
    ops._call_custom("__matmul_add_relu", out, operands)
    h4, _, _ = counters()
    assert h4 - h3 == x.nbytes
    # mode 0: everything travels every time
    lib.annc_set_operand_cache(0, 0)
    ops._call_custom("__matmul_add_relu", out, operands)
    h5, _, _ = counters()
    assert h5 - h4 == x.nbytes + w.nbytes + addend.nbytes
    assert nerr(out, oracle.matmul_add_relu(addend, x, w)) <= 2e-3


def test_output_of_one_call_is_not_uploaded_for_the_next():
    rng = np.random.default_rng(1)
    m, k, n, n2 = 200, 128, 256, 64
    x = rng.standard_normal((m, k)).astype(np.float32)
    w1 = (rng.standard_normal((k, n)) / 8).astype(np.float32)
    w2 = (rng.standard_normal((n, n2)) / 8).astype(np.float32)
    y1 = np.empty((m, n), np.float32)
    y2 = np.empty((m, n2), np.float32)
    for it in range(2):
        ops._call_custom("__matmul", y1, [x, w1, ops.shape_info(x), ops.shape_info(w1)])
        h0, _, s0 = counters()
        ops._call_custom("__matmul", y2, [y1, w2, ops.shape_info(y1), ops.shape_info(w2)])
        h1, _, s1 = counters()
        # y1 sits on the device already; w2 travels on the first round only
        assert h1 - h0 == (w2.nbytes if it == 0 else 0)
        assert s1 - s0 >= y1.nbytes
        want = oracle.matmul(oracle.matmul(x, w1), w2)
        assert nerr(y2, want) <= 4e-3
        # the host touches y1: it must travel again
        y1[3, 5] += 1.0
        y1[:] = y1 * 1.0
    y1[:] = rng.standard_normal((m, n)).astype(np.float32)
    h0, _, _ = counters()
    ops._call_custom("__matmul", y2, [y1, w2, ops.shape_info(y1), ops.shape_info(w2)])
    h1, _, _ = counters()
    assert h1 - h0 == y1.nbytes
    assert nerr(y2, oracle.matmul(y1, w2)) <= 2e-3


def test_layout_matmul_keeps_the_relaid_weight():
    rng = np.random.default_rng(2)
    m, k, n = 256, 704, 384
    x = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((k, n)) / 16).astype(np.float32)
    packed = oracle.kn4_pack(w) if hasattr(oracle, "kn4_pack") else None
    if packed is None:
        offs = oracle.kn4_offsets(k, n)
        packed = np.empty(k * n, np.float32)
        packed[offs] = w.reshape(-1)
        packed = packed.reshape(k, n)
    out = np.empty((m, n), np.float32)
    operands = [x, packed, ops.shape_info(x), ops.shape_info(packed)]
    want = oracle.layout_matmul(x, packed)
    ops._call_custom("__layout_matmul", out, operands)
    assert nerr(out, want) <= 2e-3
    h0, _, _ = counters()
    for _ in range(3):
        out[:] = 0
        ops._call_custom("__layout_matmul", out, operands)
        assert nerr(out, want) <= 2e-3
    h1, _, _ = counters()
    assert h1 - h0 == 0
    # device activations, host weight: the call has nothing to stage and does not wait
    xd = torch.from_numpy(x).cuda()
    od = torch.empty((m, n), device="cuda")
    ops._call_custom("__layout_matmul", od, [xd, packed, ops.shape_info(x), ops.shape_info(packed)])
    torch.cuda.synchronize()
    assert nerr(od.cpu().numpy(), want) <= 2e-3
    assert counters()[0] - h1 == 0


def _host_layout_matmul(x, packed):
    out = torch.empty((x.shape[0], packed.shape[1]), device="cuda")
    ops._call_custom("__layout_matmul", out, [x, packed, ops.shape_info(x), ops.shape_info(packed)])
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _host_weight(k, n):
    """Device activations of a drawn batch, a packed weight in a host buffer of its own, the weight."""
    rng = np.random.default_rng(k + n)
    w = (rng.standard_normal((k, n)) / 16).astype(np.float32)
    return lambda m: rng.standard_normal((m, k)).astype(np.float32), oracle.kn4_pack(w), w


@pytest.mark.parametrize("first", [1, 63])
def test_layout_matmul_host_weight_first_seen_by_a_small_batch(first):
    """A batch too small for the re-laid form leaves nothing behind that a larger one would take for it."""
    k, n = 512, 1028
    draw, packed, w = _host_weight(k, n)
    for m in (first, 200, first, 300):
        x = draw(m)
        got = _host_layout_matmul(torch.from_numpy(x).cuda(), packed)
        assert nerr(got, x.astype(np.float64) @ w) <= 2e-3


def test_layout_matmul_host_weight_in_both_layouts():
    """The re-laid layout goes with the batch (column tiles of a large one want [N,K]): each is kept on
    its own, and a weight of another shape in the same bytes has its own as well."""
    k, n = 2048, 1024
    draw, packed, w = _host_weight(k, n)
    for m in (8192, 200, 8192, 70):
        x = draw(m)
        got = _host_layout_matmul(torch.from_numpy(x).cuda(), packed)
        assert nerr(got, x.astype(np.float64) @ w) <= 2e-3
    other = packed.reshape(n, k)
    w2 = oracle.kn4_unpack(other, n, k)
    x = np.random.default_rng(1).standard_normal((200, n)).astype(np.float32)
    got = _host_layout_matmul(torch.from_numpy(x).cuda(), other)
    assert nerr(got, x.astype(np.float64) @ w2) <= 2e-3


def test_layout_matmul_host_weight_across_streams():
    """A stream that finds the re-laid copy of another waits for the pass that fills it."""
    k, n = 1024, 516
    draw, packed, w = _host_weight(k, n)
    _host_layout_matmul(torch.from_numpy(draw(1)).cuda(), packed)  # uploads the weight, re-lays nothing
    x = [draw(200), draw(200)]
    xd = [torch.from_numpy(a).cuda() for a in x]
    out = [torch.empty((200, n), device="cuda") for _ in x]
    torch.cuda.synchronize()
    for i, s in enumerate([torch.cuda.Stream(), torch.cuda.Stream()]):
        with torch.cuda.stream(s):
            if i == 0:
                torch.cuda._sleep(100_000_000)  # the first stream is late
            ops._use_current_stream()
            ops._call_custom("__layout_matmul", out[i], [xd[i], packed, ops.shape_info(x[i]), ops.shape_info(packed)])
    torch.cuda.synchronize()
    for a, o in zip(x, out):
        assert nerr(o.cpu().numpy(), a.astype(np.float64) @ w) <= 2e-3


def test_layout_matmul_constant_registered_again():
    """A registered weight whose contents change is registered again: its re-laid copy follows."""
    k, n = 352, 260
    draw, packed, w = _host_weight(k, n)
    x = draw(200)
    try:
        for scale in (1.0, -3.0):
            packed[:] = oracle.kn4_pack((scale * w).astype(np.float32))
            assert lib.annc_register_constant(packed.ctypes.data, packed.nbytes) == 0
            got = _host_layout_matmul(torch.from_numpy(x).cuda(), packed)
            assert nerr(got, scale * (x.astype(np.float64) @ w)) <= 2e-3
    finally:
        assert lib.annc_unregister_constant(packed.ctypes.data) == 0


@pytest.mark.parametrize("cap", [1, 1 << 20])
def test_operands_beyond_the_cap_are_kept_for_their_call(cap):
    """A call whose operands do not fit under the cap has them all on the device until it ends; the next
    one uploads what was dropped since."""
    rng = np.random.default_rng(4)
    lib.annc_set_operand_cache(2, cap)
    try:
        for m, k, n in ((300, 512, 1024), (70, 2048, 516), (300, 512, 1024)):
            x = rng.standard_normal((m, k)).astype(np.float32)
            w = (rng.standard_normal((k, n)) / 16).astype(np.float32)
            addend = rng.standard_normal((m, n)).astype(np.float32)
            out = np.empty((m, n), np.float32)
            info = [ops.shape_info(addend), ops.shape_info(addend), ops.shape_info(x), ops.shape_info(w)]
            ops._call_custom("__matmul_add_relu", out, [addend, addend, x, w] + info)
            assert nerr(out, oracle.matmul_add_relu(addend, x, w)) <= 2e-3
            packed = oracle.kn4_pack(w)
            ops._call_custom("__layout_matmul", out, [x, packed, ops.shape_info(x), ops.shape_info(packed)])
            assert nerr(out, x.astype(np.float64) @ w) <= 2e-3
    finally:
        lib.annc_set_operand_cache(2, 24 << 30)


def test_a_wait_that_ran_out_is_reported(capfd):
    rng = np.random.default_rng(3)
    a = rng.standard_normal((256, 256)).astype(np.float32)
    b = rng.standard_normal((256, 256)).astype(np.float32)
    out = np.empty((256, 256), np.float32)
    try:
        assert lib.annc_gemm_debug_set_error_word(1) == 0
        ops._call_custom("__matmul", out, [a, b, ops.shape_info(a), ops.shape_info(b)])
        assert "wait ran out" in lib.annc_last_error().decode()
        assert "__matmul failed" in capfd.readouterr().err
    finally:
        assert lib.annc_gemm_debug_set_error_word(0) == 0
    ops._call_custom("__matmul", out, [a, b, ops.shape_info(a), ops.shape_info(b)])
    assert nerr(out, oracle.matmul(a, b)) <= 2e-3
