"""Parity of the GEMM custom calls, kernel-selector entry points and the
KPFusedBatchMatMulAddSigmoid twin with the CPU oracle, through the C ABI.
Error measure: normwise max|y - ref| / max|ref| against the fp32 OpenBLAS result;
bound 2e-3 for the TF32 tensor-core route, 1e-2 for BF16, 2e-5 for the fp32 route."""
import numpy as np
import pytest

from oracle import oracle
from tests.golden import reference_cases as rc

pytestmark = pytest.mark.gpu

import torch
from annc_b200 import ops  # noqa: E402  (no fallback: a missing library fails the collection)
from annc_b200 import AnncError, _lib, device, synth  # noqa: E402

TOL = {"simt_fp32": 2e-5, "tcgen05_tf32": 2e-3, "tcgen05_pair_tf32": 2e-3, "tcgen05_pair_bf16": 1e-2}


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def nerr(got, want):
    got = got.cpu().numpy() if hasattr(got, "cpu") else got
    return float(np.abs(got - want).max() / max(np.abs(want).max(), 1e-30))


def _tol_for(m, n, k, **kw):
    d = _lib.GemmDesc()
    d.m, d.n, d.k, d.batch = m, n, k, kw.get("batch", 1)
    d.lda, d.ldb, d.ldc = k, n, n
    d.stride_a, d.stride_b, d.stride_c = m * k, k * n, m * n
    d.a = d.b = d.c = 256  # alignment probe only
    d.trans_a, d.trans_b = int(kw.get("trA", False)), int(kw.get("trB", False))
    d.b_format = kw.get("b_format", 0)
    return TOL[_lib.lib.annc_gemm_kernel_name(__import__("ctypes").byref(d)).decode()]


@pytest.mark.parametrize("shape", [(12, 12, 12), (13, 17, 19), (64, 64, 64), (100, 130, 77),
                                   (128, 128, 128), (256, 512, 384), (512, 1024, 1024),
                                   (1000, 520, 264), (129, 257, 100)])
@pytest.mark.parametrize("where", ["host", "device"])
def test_matmul_custom_call(shape, where):
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    want = oracle.matmul(a, b)
    got = ops.xla_matmul(_dev(a), _dev(b)) if where == "device" else ops.xla_matmul(a, b)
    assert nerr(got, want) <= _tol_for(m, n, k)


def test_matmul_add_relu_config():
    """BASELINE config: X[512,1024] ~ U(-1,1), W[1024,1024] ~ N(0,1/32), bias ~ N(0,0.1)."""
    x, w, bias, addend, maxop = synth.matmul_add_relu_case(0)
    want = oracle.matmul_add_relu(addend, x, w)
    got = ops.xla_matmul_add_relu(_dev(maxop), _dev(addend), _dev(x), _dev(w))
    assert nerr(got, want) <= _tol_for(512, 1024, 1024)
    assert (got.cpu().numpy() >= 0).all()
    got_add = ops.xla_matmul_add(addend, x, w)
    assert nerr(got_add, oracle.matmul_add(addend, x, w)) <= _tol_for(512, 1024, 1024)


@pytest.mark.parametrize("shape", [(4, 16, 8, 24), (64, 256, 64, 256), (3, 27, 64, 27), (70000, 8, 8, 8)])
def test_batch_matmul_custom_call(shape):
    b, m, k, n = shape
    rng = np.random.default_rng(b)
    A = rng.standard_normal((b, m, k)).astype(np.float32)
    B = rng.standard_normal((b, k, n)).astype(np.float32)
    got = ops.xla_batch_matmul(_dev(A), _dev(B))
    assert nerr(got, oracle.batch_matmul(A, B)) <= _tol_for(m, n, k, batch=b)


@pytest.mark.parametrize("shape", [(12, 12, 12), (40, 30, 20), (64, 353, 129), (128, 400, 140),
                                   (256, 705, 257), (512, 1024, 1024)])
def test_layout_matmul_custom_call(shape):
    m, k, n = shape
    rng = np.random.default_rng(k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = rng.standard_normal((k, n)).astype(np.float32)
    packed = oracle.kn4_pack(w)  # pinned to the reference packer in the CPU tests
    want = oracle.layout_matmul(a, packed)
    got = ops.xla_layout_matmul(_dev(a), _dev(packed))
    assert nerr(got, want) <= _tol_for(m, n, k, b_format=1)


def test_kn4_device_pack_unpack_bit_exact():
    for K, N in [(12, 12), (353, 129), (705, 257), (2048, 4096)]:
        w = np.arange(K * N, dtype=np.float32).reshape(K, N)
        packed = device.kn4_pack(_dev(w))
        if K * N < 1_000_000:
            np.testing.assert_array_equal(packed.cpu().numpy(), oracle.kn4_pack(w))
        assert torch.equal(device.kn4_unpack(packed), _dev(w))
    offs = oracle.kn4_offsets(705, 257)
    for k, n in [(0, 0), (704, 256), (352, 128), (351, 127), (500, 200)]:
        assert _lib.lib.annc_kn4_offset(705, 257, k, n) == offs[k, n]


@pytest.mark.parametrize("variant", ["Sequential", "Parallel", "MLIR"])
@pytest.mark.parametrize("trA,trB", [(False, False), (True, False), (False, True), (True, True)])
def test_selector_gemm(variant, trA, trB):
    M, N, K = 70, 50, 90
    rng = np.random.default_rng(1)
    A = rng.standard_normal((K, M) if trA else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if trB else (K, N)).astype(np.float32)
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    for alpha, beta in [(1.0, 0.0), (0.5, 1.0), (2.0, -0.25)]:
        want = oracle.sgemm(trA, trB, A, B, M, N, K, alpha, beta, C0)
        got = ops.selector_gemm(variant, trA, trB, A, B, M, N, K, alpha, beta, C0)
        assert nerr(got, want) <= 2e-5


def test_selector_empty_variants_are_noops():
    A = np.ones((4, 4), np.float32)
    C0 = np.full((4, 4), 3.0, np.float32)
    got = ops.selector_gemm("Empty", False, False, A, A, 4, 4, 4, 1.0, 0.0, C0)
    np.testing.assert_array_equal(got, C0)


@pytest.mark.parametrize("trB", [False, True])
def test_selector_batch3d_4d(trB):
    rng = np.random.default_rng(4)
    P, Q, M, N, K = 6, 2, 26, 4, 26
    A = rng.standard_normal((Q, P, M, K)).astype(np.float32)
    B = rng.standard_normal((Q, P, N, K) if trB else (Q, P, K, N)).astype(np.float32)
    Bm = np.swapaxes(B, -1, -2) if trB else B
    want = np.matmul(A, Bm)
    got4 = ops.selector_batch4d("Sequential", False, trB, A, B, Q, P, M, N, K)
    assert nerr(got4, want) <= 2e-5
    got3 = ops.selector_batch3d("Parallel", False, trB, A[0], B[0], P, M, N, K)
    assert nerr(got3, want[0]) <= 2e-5


@pytest.mark.parametrize("trA", [False, True])
def test_selector_gemv(trA):
    rng = np.random.default_rng(8)
    M, N = 300, 77
    A = rng.standard_normal((M, N)).astype(np.float32)
    X = rng.standard_normal(M if trA else N).astype(np.float32)
    Y0 = rng.standard_normal(N if trA else M).astype(np.float32)
    for alpha, beta in [(1.0, 0.0), (0.5, 2.0)]:
        want = oracle.sgemv(trA, A, X, M, N, alpha, beta, Y0)
        got = ops.selector_gemv("", trA, A, X, M, N, alpha, beta, Y0)
        assert nerr(got, want) <= 2e-5


@pytest.mark.parametrize("case", rc.BMM_ADD_SIGMOID, ids=lambda c: c["name"])
def test_bmm_add_sigmoid_golden(case):
    lhs, rhs, bias = rc.bmm_case_tensors(case)
    want = rc.bmm_reference(lhs, rhs, bias)
    got = ops.kp_fused_batch_matmul_add_sigmoid(lhs, rhs, bias)
    np.testing.assert_allclose(got, want, atol=1e-5, rtol=0)  # tolerance of the reference test
    got_d = ops.kp_fused_batch_matmul_add_sigmoid(_dev(lhs), _dev(rhs), _dev(bias))
    np.testing.assert_allclose(got_d.cpu().numpy(), want, atol=1e-5, rtol=0)


@pytest.mark.parametrize("err", rc.BMM_ADD_SIGMOID_ERRORS, ids=lambda e: e[3][:20])
def test_bmm_add_sigmoid_errors(err):
    ls, rs, bs, msg = err
    with pytest.raises(AnncError) as e:
        ops.kp_fused_batch_matmul_add_sigmoid(np.zeros(ls, np.float32), np.zeros(rs, np.float32),
                                              np.zeros(bs, np.float32))
    assert msg in e.value.message


@pytest.mark.parametrize("m,n,k", [(4096, 512, 13), (1500, 64, 16), (1024, 8, 1)])
def test_small_k_route(m, n, k):
    """First DLRM layer shape class: k <= 16, bias + ReLU, fp32 exact route."""
    rng = np.random.default_rng(k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    c = torch.empty((m, n), device="cuda")
    name = device.gemm(_dev(a), _dev(b), c, m=m, n=n, k=k, bias=_dev(bias), activation=1)
    want = np.maximum(a @ b + bias, 0)
    assert name == "simt_fp32"
    assert nerr(c, want) <= 2e-5


@pytest.mark.parametrize("shared_b", [False, True])
@pytest.mark.parametrize("trans_b", [False, True])
def test_strided_batch_on_tensor_cores(shared_b, trans_b):
    """Strided-batch GEMM through rank-3 tensor maps (tails in m, n and k inside every batch)."""
    b, m, n, k = 5, 200, 136, 100
    rng = np.random.default_rng(7)
    A = rng.standard_normal((b, m, k)).astype(np.float32)
    B = rng.standard_normal((1 if shared_b else b, k, n)).astype(np.float32)
    want = np.matmul(A, B)
    Bd = _dev(np.swapaxes(B, 1, 2)) if trans_b else _dev(B)
    c = torch.full((b, m, n), float("nan"), device="cuda")
    name = device.gemm(_dev(A), Bd, c, m=m, n=n, k=k, batch=b, trans_b=trans_b, stride_a=m * k,
                       stride_b=0 if shared_b else k * n, stride_c=m * n)
    assert name in ("tcgen05_tf32", "tcgen05_pair_tf32") and not device.gemm_timed_out()
    assert nerr(c, want) <= 2e-3


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (1, 33, 512), (31, 32, 33), (33, 31, 128), (63, 260, 1000), (64, 65, 31),
                                   (65, 64, 17), (70, 2000, 96), (1000, 1030, 20), (65, 64, 16), (130, 516, 13),
                                   (64, 4, 1), (1001, 8, 8)])
@pytest.mark.parametrize("trA,trB,kn4", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1), (1, 0, 1)])
def test_fp32_route_tile_edges(m, n, k, trA, trB, kn4):
    """The fp32 tiles at their edges, both loads (16-byte and one float at a time), every operand
    order and K split over a cluster.  Bound: a chain of k rounded multiply-adds, and three more
    roundings for alpha, beta * C and bias, is within (k + 4) ulp of the sum of magnitudes."""
    rng = np.random.default_rng(m + 3 * n + 7 * k + trA)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    c0 = rng.standard_normal((m, n)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    bd = oracle.kn4_pack(b) if kn4 else (b.T if trB else b)
    c = _dev(c0)
    name = device.gemm(_dev(a.T if trA else a), _dev(bd), c, m=m, n=n, k=k, trans_a=bool(trA), trans_b=bool(trB),
                       alpha=0.5, beta=2.0, bias=_dev(bias), b_format=_lib.B_KN4 if kn4 else _lib.B_PLAIN,
                       math=_lib.MATH_FP32)
    assert name == "simt_fp32"
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    want = 0.5 * (a64 @ b64) + 2.0 * c0 + bias
    size = 0.5 * (abs(a64) @ abs(b64)) + 2.0 * abs(c0) + abs(bias)
    assert (abs(c.cpu().numpy() - want) <= (k + 4) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("bias_shape", [(1,), (24,), (1, 24), (50, 1), (50, 24), (7, 1, 1), (7, 50, 24), (1, 1, 24)])
@pytest.mark.parametrize("batched", [False, True])
def test_batch_matmul_add_sigmoid_bias_broadcast(bias_shape, batched):
    """A shared right-hand side is multiplied as one tall product when the bias allows it."""
    rng = np.random.default_rng(len(bias_shape))
    lhs = rng.standard_normal((7, 50, 36)).astype(np.float32)
    rhs = rng.standard_normal((7, 36, 24) if batched else (36, 24)).astype(np.float32)
    bias = rng.standard_normal(bias_shape).astype(np.float32)
    got = ops.kp_fused_batch_matmul_add_sigmoid(_dev(lhs), _dev(rhs), _dev(bias)).cpu().numpy()
    want = 1 / (1 + np.exp(-(np.matmul(lhs.astype(np.float64), rhs.astype(np.float64)) + bias)))
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("m,n,k", [(64, 16, 32), (200, 140, 352), (300, 264, 353), (130, 4100, 100), (70, 260, 1061),
                                   (2100, 1000, 704)])
def test_layout_matmul_device_weight(m, n, k):
    """A packed weight on the device is re-laid into scratch by each call (K chunks of 352 and the two
    that share the rest, panels of 12 and 4 columns, tiles of 128 x 32)."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k), device="cuda", generator=g)
    w = torch.randn((k, n), device="cuda", generator=g)
    packed = device.kn4_pack(w)
    np.testing.assert_array_equal(packed.cpu().numpy(), oracle.kn4_pack(w.cpu().numpy()))
    assert torch.equal(device.kn4_unpack(packed), w)
    got = ops.xla_layout_matmul(a, packed)
    want = (a.double() @ w.double()).cpu().numpy()
    assert nerr(got, want) <= 2e-3  # TF32


@pytest.mark.parametrize("off", [1, 2, 3])
def test_layout_matmul_device_weight_off_16_bytes(off):
    """A packed weight that is a view at an odd place of a larger buffer."""
    g = torch.Generator(device="cuda").manual_seed(off)
    m, k, n = 200, 356, 264
    a = torch.randn((m, k), device="cuda", generator=g)
    w = torch.randn((k, n), device="cuda", generator=g)
    packed = torch.empty(k * n + off, device="cuda")[off:].view(k, n).copy_(device.kn4_pack(w))
    assert packed.data_ptr() % 16 == 4 * off
    got = ops.xla_layout_matmul(a, packed)
    want = (a.double() @ w.double()).cpu().numpy()
    assert nerr(got, want) <= 2e-5  # the fp32 route


def test_layout_matmul_device_weight_streams_and_capture():
    """The scratch is safe across streams of a thread, and a captured call does without it."""
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn((256, 512), device="cuda", generator=g)
    packed = [device.kn4_pack(torch.randn((512, 768), device="cuda", generator=g)) for _ in range(2)]
    want = [ops.xla_layout_matmul(a, p) for p in packed]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for i in range(40):
        with torch.cuda.stream(streams[i % 2]):
            outs.append(ops.xla_layout_matmul(a, packed[i % 2]))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = ops.xla_layout_matmul(a, packed[0])
    graph.replay()
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        assert torch.equal(o, want[i % 2])
    assert nerr(captured, want[0].cpu().numpy()) <= 1e-5  # the same products, summed in another tiling


@pytest.mark.parametrize("k", range(1, 18))
@pytest.mark.parametrize("m,n", [(64, 4), (79, 516)])
def test_small_k_product_at_every_k(m, n, k):
    """Bias, ReLU and beta * C, with ragged rows.  Bound: a chain of k rounded multiply-adds and three more
    roundings."""
    rng = np.random.default_rng(k + n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    c0, bias = rng.standard_normal((m, n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    c = _dev(c0)
    device.gemm(_dev(a), _dev(b), c, m=m, n=n, k=k, beta=-1.0, bias=_dev(bias), activation=1, math=_lib.MATH_FP32)
    want = np.maximum(a.astype(np.float64) @ b - c0 + bias, 0)
    size = abs(a).astype(np.float64) @ abs(b) + abs(c0) + abs(bias)
    assert (abs(c.cpu().numpy() - want) <= (k + 4) * 2.0 ** -24 * size).all()


def test_a_call_without_scratch_does_not_wait_for_one_with():
    """Calls of one thread on two streams: only those that take the thread's scratch follow each other."""
    g = torch.Generator(device="cuda").manual_seed(10)
    a, w = torch.randn((200, 512), device="cuda", generator=g), torch.randn((512, 1000), device="cuda", generator=g)
    packed, x = device.kn4_pack(w), torch.randn((64, 64), device="cuda", generator=g)
    want = [ops.xla_layout_matmul(a, packed), ops.xla_matmul(x, x)]
    torch.cuda.synchronize()
    late, other = torch.cuda.Stream(), torch.cuda.Stream()
    done = torch.cuda.Event()
    with torch.cuda.stream(late):
        torch.cuda._sleep(400_000_000)
        first = ops.xla_layout_matmul(a, packed)
    with torch.cuda.stream(other):
        plain = ops.xla_matmul(x, x)
        done.record(other)
        done.synchronize()
        assert not late.query()
        second = ops.xla_layout_matmul(a, packed)  # waits for the scratch
        other.synchronize()
        assert late.query()
    assert torch.equal(plain, want[1]) and torch.equal(first, want[0]) and torch.equal(second, want[0])


def test_layout_matmul_beside_a_capture_of_another_thread():
    """A thread whose first call takes scratch, and that ends and gives it back, while another thread
    captures: the capture goes on."""
    import threading
    g = torch.Generator(device="cuda").manual_seed(9)
    a = torch.randn((200, 512), device="cuda", generator=g)
    w = torch.randn((512, 1000), device="cuda", generator=g)
    packed, out = device.kn4_pack(w), torch.empty((200, 1000), device="cuda")
    x, y = torch.randn((64, 64), device="cuda", generator=g), torch.empty((64, 64), device="cuda")
    step = lambda: device.gemm(x, x, y, m=64, n=64, k=64)
    step()
    ops.xla_layout_matmul(a, packed)  # the kernels are loaded
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def other():
        with torch.cuda.stream(streams[1]):
            ops._call_custom("__layout_matmul", out, [a, packed, ops.shape_info(a), ops.shape_info(packed)])

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        step()
        t = threading.Thread(target=other)
        t.start()
        t.join()
        step()
    y.fill_(-7.0)
    graph.replay()
    torch.cuda.synchronize()
    assert nerr(y, (x.double() @ x.double()).cpu().numpy()) <= 2e-3
    assert nerr(out, (a.double() @ w.double()).cpu().numpy()) <= 2e-3


@pytest.mark.parametrize("m,n", [(64, 128), (200, 512), (2048, 512), (20000, 256), (4096, 1)])
def test_back_to_back_products_wait_for_each_other(m, n):
    """Kernels that are launched while the one before them drains read what that one wrote and overwrite what it
    read: a chain of products over two buffers is the same, bit for bit, with the device idle between them."""
    g = torch.Generator(device="cuda").manual_seed(m)
    w = torch.randn((512, 512), device="cuda", generator=g) * 512 ** -0.5
    last = torch.randn((512, n), device="cuda", generator=g) * 512 ** -0.5
    bias, tail = torch.randn(512, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g)
    x0 = torch.randn((m, 512), device="cuda", generator=g)

    def chain(wait):
        x, y, out = x0.clone(), torch.empty_like(x0), []
        for _ in range(12):
            for a, b in ((x, y), (y, x)):
                device.gemm(a, w, b, m=m, n=512, k=512, bias=bias, activation=1)
                if wait:
                    torch.cuda.synchronize()
            out.append(torch.empty((m, n), device="cuda"))
            device.gemm(x, last, out[-1], m=m, n=n, k=512, bias=tail)
            if wait:
                torch.cuda.synchronize()
        return out + [x]

    for a, b in zip(chain(False), chain(True)):
        assert torch.equal(a, b)


def _same_with_and_without_waiting(chain):
    """chain(wait) calls wait() after each of its steps; its outputs are those of the run that waits each time."""
    want = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    for _ in range(3):
        got = chain(lambda: None)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("m,bf16", [(128, False), (512, False), (1024, False), (4096, False), (256, True), (4096, True)])
def test_a_product_reads_what_the_one_before_it_wrote(m, bf16):
    """... as its A, its B, its bias or its addend, and overwrites what that one read: kernels of both tile sizes and of
    split K, which are launched while the one before them drains."""
    g = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=g)
    n = k = 512
    a0, b0, t0, add0 = rnd(m, k), rnd(k, n) * k ** -0.5, rnd(n, n) * n ** -0.5, rnd(m, n)
    bias0 = rnd(n)
    if bf16:
        a0, b0, t0 = a0.bfloat16(), (b0.t().contiguous()).bfloat16(), t0.bfloat16()

    def chain(wait):
        a, b, bias, add = a0.clone(), b0.clone(), bias0.clone(), add0.clone()
        out = []

        def mul(x, y, c, rows, **kw):
            if bf16:
                flags = _lib.IO_A_BF16 | _lib.IO_B_BF16 | (_lib.IO_C_BF16 if c.dtype is torch.bfloat16 else 0)
                kw.update(trans_b=True, math=_lib.MATH_BF16, io_flags=flags)
            device.gemm(x, y, c, m=rows, n=n, k=k, **kw)
            wait()

        for _ in range(6):
            c = torch.empty((m, n), device="cuda")
            nb = torch.empty_like(b)
            mul(t0, b, nb, n)  # the next product's B ...
            row = torch.empty((256, n), device="cuda")
            mul(a[:128].repeat(2, 1), nb, row, 256, activation=1)  # ... and from it a bias
            full = torch.empty((m, n), device="cuda")
            mul(a, nb, full, m, addend=add, bias=row[3])
            mul(a, b, c, m, addend=full, bias=row[5], activation=1)  # the addend of the launch before
            mul(a, nb, full, m, bias=bias)  # over what that one read
            bias = row[7]
            na = torch.empty_like(a)
            mul(a, b, na, m)
            mul(na, nb, c, m, addend=full)
            a, add = na, full
            out += [c.clone(), full.clone(), row.clone()]
        return out

    _same_with_and_without_waiting(chain)


@pytest.mark.parametrize("batch", [1, 100, 3000, 20000])
def test_interaction_between_products(batch):
    """z is written by the product before the interaction, what it wrote is read by the one behind it, and the next
    round's first product overwrites z."""
    g = torch.Generator(device="cuda").manual_seed(batch)
    F, D, H, pad = 27, 64, 256, 416
    x0 = torch.randn((batch, H), device="cuda", generator=g)
    w = torch.randn((H, D), device="cuda", generator=g) * H ** -0.5
    top = torch.randn((pad, H), device="cuda", generator=g) * pad ** -0.5
    last = torch.randn((H, 1), device="cuda", generator=g) * H ** -0.5
    z0 = torch.randn((batch, F, D), device="cuda", generator=g)

    def chain(wait):
        x, z, inter, out = x0.clone(), z0.clone(), torch.full((batch, pad), -3.0, device="cuda"), []
        for _ in range(8):
            device.gemm(x, w, z, m=batch, n=D, k=H, ldc=F * D, activation=1)
            wait()
            device.dot_interaction(z, inter)
            wait()
            device.gemm(inter, top, x, m=batch, n=H, k=pad, activation=1)
            wait()
            out.append(torch.empty((batch, 1), device="cuda"))
            device.gemm(x, last, out[-1], m=batch, n=1, k=H, activation=2)
            wait()
        return out + [x, z, inter]

    _same_with_and_without_waiting(chain)


@pytest.mark.parametrize("m,n", [(64, 128), (20000, 512), (64, 1)])
def test_a_refused_launch_is_reported_once(m, n):
    """A product on a stream whose capture was ended by an error is refused; the one after it runs."""
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    x, w = torch.randn((m, 128), device="cuda"), torch.randn((128, n), device="cuda")
    y = torch.empty((m, n), device="cuda")
    stream = torch.cuda.Stream()
    handle, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    call = lambda: device.gemm(x, w, y, m=m, n=n, k=128, stream=stream.cuda_stream)
    call()
    stream.synchronize()
    assert rt.cudaStreamBeginCapture(handle, 1) == 0  # of this thread only
    assert rt.cudaStreamSynchronize(handle) != 0  # not permitted now: the capture is over
    with pytest.raises(AnncError):
        call()
    assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0 and not graph
    rt.cudaGetLastError()
    call()
    stream.synchronize()
    assert nerr(y, (x.double() @ w.double()).cpu().numpy()) <= 2e-3
