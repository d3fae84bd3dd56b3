"""The persistent CTA-pair tcgen05 GEMM (TF32 and BF16) against the fp32 OpenBLAS oracle:
both B layouts, tails in M, N and K, every epilogue, strided batches, bf16 output and the
fused row softmax.  Bounds (normwise max|y - ref| / max|ref|): 2e-3 TF32, 1e-2 BF16;
softmax 1e-5 absolute on the probabilities of TF32-rounded logits is not meaningful, so the
fused softmax is compared with the softmax of this kernel's own logits (1e-6) and with the
oracle's probabilities within the TF32 bound."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

import torch
import annc_b200  # noqa: F401,E402  (no fallback: a missing library fails the collection)
from annc_b200 import device  # noqa: E402
from annc_b200._lib import (ACT_NONE, ACT_RELU, ACT_SIGMOID, IO_A_BF16, IO_B_BF16, IO_C_BF16,  # noqa: E402
                            IO_PAIR, IO_SOFTMAX, MATH_BF16, MATH_TF32)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def nerr(got, want):
    return float(np.abs(got.float().cpu().numpy() - want).max() / np.abs(want).max())


SHAPES = [(256, 256, 32), (256, 256, 256), (512, 512, 96), (300, 200, 100), (1000, 520, 264),
          (257, 192, 36), (2048, 1024, 1024), (4096, 512, 416), (640, 768, 2048), (8192, 256, 64)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("bsrc", ["nk", "kn"])
def test_pair_tf32(m, n, k, bsrc):
    rng = np.random.default_rng(m + 7 * n + 13 * k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    want = oracle.matmul(a, b)
    c = torch.full((m, n), float("nan"), device="cuda")
    if bsrc == "nk":
        name = device.gemm(_dev(a), _dev(b.T), c, m=m, n=n, k=k, trans_b=True, math=MATH_TF32, io_flags=IO_PAIR)
    else:
        name = device.gemm(_dev(a), _dev(b), c, m=m, n=n, k=k, math=MATH_TF32, io_flags=IO_PAIR)
    assert name == "tcgen05_pair_tf32"
    assert not device.gemm_timed_out()
    assert nerr(c, want) <= 2e-3


@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_SIGMOID])
@pytest.mark.parametrize("with_addend,with_bias,alpha,beta", [(False, True, 1.0, 0.0), (True, False, 1.0, 0.0),
                                                              (True, True, 0.5, 2.0), (False, False, 2.0, -1.0)])
def test_pair_epilogues(act, with_addend, with_bias, alpha, beta):
    m, n, k = 600, 328, 96
    rng = np.random.default_rng(act + 10)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    c0 = rng.standard_normal((m, n)).astype(np.float32)
    add = rng.standard_normal((m, n)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    pre = alpha * (a @ b) + beta * c0
    want = pre.copy()
    if with_addend:
        want = want + add
    if with_bias:
        want = want + bias
    if act == ACT_RELU:
        want = np.maximum(want, 0)
    elif act == ACT_SIGMOID:
        want = 1 / (1 + np.exp(-want))
    c = _dev(c0)
    name = device.gemm(_dev(a), _dev(b), c, m=m, n=n, k=k, alpha=alpha, beta=beta,
                       addend=_dev(add) if with_addend else None, bias=_dev(bias) if with_bias else None,
                       activation=act, math=MATH_TF32, io_flags=IO_PAIR)
    assert name == "tcgen05_pair_tf32" and not device.gemm_timed_out()
    assert np.abs(c.cpu().numpy() - want).max() <= 2e-3 * np.abs(pre).max()


def test_pair_strided_batch_and_pitched_output():
    bsz, m, n, k = 5, 300, 256, 64
    rng = np.random.default_rng(2)
    a = rng.standard_normal((bsz, m, k)).astype(np.float32)
    b = rng.standard_normal((bsz, k, n)).astype(np.float32)
    want = np.matmul(a, b)
    c = torch.full((bsz, m, n + 8), 9.0, device="cuda")
    name = device.gemm(_dev(a), _dev(b), c, m=m, n=n, k=k, batch=bsz, stride_a=m * k, stride_b=k * n,
                       stride_c=m * (n + 8), ldc=n + 8, math=MATH_TF32, io_flags=IO_PAIR)
    assert name == "tcgen05_pair_tf32" and not device.gemm_timed_out()
    got = c.cpu().numpy()
    assert (got[:, :, n:] == 9.0).all()
    assert np.abs(got[:, :, :n] - want).max() <= 2e-3 * np.abs(want).max()


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (1000, 520, 264), (4096, 1024, 8192), (8192, 64, 512)])
@pytest.mark.parametrize("c_bf16", [False, True])
def test_pair_bf16(m, n, k, c_bf16):
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = (rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    want = np.maximum(oracle.matmul(a, b) + bias, 0)
    a16 = device.cast_bf16(_dev(a))
    b16 = device.bf16_weight(_dev(b))
    assert torch.equal(a16, _dev(a).to(torch.bfloat16)) and torch.equal(b16, _dev(b).t().contiguous().to(torch.bfloat16))
    c = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16 if c_bf16 else torch.float32)
    flags = IO_A_BF16 | IO_B_BF16 | (IO_C_BF16 if c_bf16 else 0)
    name = device.gemm(a16, b16, c, m=m, n=n, k=k, trans_b=True, bias=_dev(bias), activation=ACT_RELU,
                       math=MATH_BF16, io_flags=flags)
    assert name == "tcgen05_pair_bf16" and not device.gemm_timed_out()
    assert nerr(c, want) <= 1e-2


@pytest.mark.parametrize("n", [256, 100])
def test_pair_batch_matmul_softmax(n):
    """batch_matmul Q K^T followed by the row softmax in one kernel."""
    bsz, m, k = 8, 256, 64
    rng = np.random.default_rng(n)
    q = (rng.standard_normal((bsz, m, k)) / 8).astype(np.float32)
    kt = rng.standard_normal((bsz, k, n)).astype(np.float32)
    logits = torch.empty((bsz, m, n), device="cuda")
    probs = torch.full((bsz, m, n), float("nan"), device="cuda")
    kw = dict(m=m, n=n, k=k, batch=bsz, stride_a=m * k, stride_b=k * n, stride_c=m * n, math=MATH_TF32)
    device.gemm(_dev(q), _dev(kt), logits, io_flags=IO_PAIR, **kw)
    name = device.gemm(_dev(q), _dev(kt), probs, io_flags=IO_SOFTMAX, **kw)
    assert name == "tcgen05_pair_tf32" and not device.gemm_timed_out()
    own = oracle.softmax(logits.cpu().numpy().reshape(-1, n)).reshape(bsz, m, n)
    assert np.abs(probs.cpu().numpy() - own).max() <= 1e-6
    ref = oracle.softmax(np.matmul(q, kt).reshape(-1, n)).reshape(bsz, m, n)
    assert np.abs(probs.cpu().numpy() - ref).max() <= 2e-3


@pytest.mark.parametrize("m,n,k,ldc,batch", [(1, 8, 32, 8, 1), (31, 40, 64, 48, 1), (257, 64, 256, 1728, 1),
                                             (300, 200, 64, 200, 3), (129, 255, 96, 260, 1), (513, 600, 36, 601, 1),
                                             (1500, 264, 512, 264, 1)])
@pytest.mark.parametrize("dt", ["tf32", "bf16", "bf16_out"])
@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU])
def test_pair_store_edges(m, n, k, ldc, batch, dt, act):
    """Epilogue with TMA stores at the edges of its 32-row chunks, with padded rows that must stay
    untouched and, where a row is not made of whole 16-byte pieces, its general form.  Against fp64: products
    of operands cut to 11 (TF32) or rounded to 8 bits, hence 2e-3 / 1e-2 of the largest value."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((batch, m, k), device="cuda", generator=g)
    b = torch.randn((batch, n, k), device="cuda", generator=g)
    bias = torch.randn(n, device="cuda", generator=g)
    io, math = IO_PAIR, MATH_TF32
    if dt != "tf32":
        if k % 8:
            pytest.skip("bf16 rows of 16 bytes")
        a, b = a.bfloat16(), b.bfloat16()
        io, math = IO_A_BF16 | IO_B_BF16 | (IO_C_BF16 if dt == "bf16_out" else 0), MATH_BF16
    c = torch.full((batch, m, ldc), -7.0, device="cuda", dtype=torch.bfloat16 if dt == "bf16_out" else torch.float32)
    device.gemm(a, b, c, m=m, n=n, k=k, batch=batch, trans_b=True, ldc=ldc, stride_a=m * k, stride_b=n * k,
                stride_c=m * ldc, alpha=0.5, bias=bias, activation=act, math=math, io_flags=io)
    assert not device.gemm_timed_out()
    want = 0.5 * (a.double() @ b.double().transpose(1, 2)) + bias
    want = want.relu() if act == ACT_RELU else want
    assert nerr(c[:, :, :n], want.float().cpu().numpy()) <= (2e-3 if dt == "tf32" else 1e-2)
    assert (c[:, :, n:] == -7.0).all()


@pytest.mark.parametrize("m,n,k,batch", [(256, 256, 64, 1), (300, 600, 96, 1), (2600, 500, 128, 1), (9500, 500, 160, 2),
                                         (19200, 260, 64, 1), (256, 129, 64, 5), (256, 140, 2048, 80)])
@pytest.mark.parametrize("form", ["nk", "kn", "bf16", "add"])
def test_pair_half_tiles(m, n, k, batch, form):
    """Tiles of a last round cut in column halves (a half beyond N, a ragged N in either half, whole
    rounds before them), in every operand form and with beta * C (the general epilogue).  Bounds as
    in test_pair_store_edges."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((batch, m, k), device="cuda", generator=g)
    b = torch.randn((batch, k, n), device="cuda", generator=g)
    c = torch.randn((batch, m, n), device="cuda", generator=g)
    add = torch.randn((batch, m, n), device="cuda", generator=g) if form == "add" else None
    if form in ("kn", "add") and n % 4:
        pytest.skip("[K,N] rows of 16 bytes")
    if form == "bf16":
        a, b = a.bfloat16(), b.bfloat16()
    beta = 0.0 if form in ("add", "bf16") else 1.0
    want = a.double() @ b.double() + beta * c.double() + (0 if add is None else add.double())
    bop = b if form in ("kn", "add") else b.transpose(1, 2).contiguous()
    device.gemm(a, bop, c, m=m, n=n, k=k, batch=batch, trans_b=form not in ("kn", "add"), stride_a=m * k,
                stride_b=n * k, stride_c=m * n, addend=add, stride_addend=m * n if add is not None else 0, beta=beta,
                math=MATH_BF16 if form == "bf16" else MATH_TF32,
                io_flags=IO_A_BF16 | IO_B_BF16 if form == "bf16" else IO_PAIR)
    assert not device.gemm_timed_out()
    assert nerr(c, want.float().cpu().numpy()) <= (1e-2 if form == "bf16" else 2e-3)


@pytest.mark.parametrize("n,m,batch", [(256, 256, 2), (130, 257, 1), (33, 100, 3)])
@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_SIGMOID])
@pytest.mark.parametrize("terms", ["", "bias", "addend", "beta", "all"])
def test_pair_softmax_terms(n, m, batch, act, terms):
    """Row softmax over act(alpha * A B + beta * C + addend + bias), at row and column remainders.  Against
    fp64: the products are off by 2^-9 of their size (operands cut to 11 bits), a softmax value by at
    most twice that error of its exponent."""
    g = torch.Generator(device="cuda").manual_seed(n + m)
    k = 64
    a = torch.randn((batch, m, k), device="cuda", generator=g) / 8
    b = torch.randn((batch, n, k), device="cuda", generator=g) / 8
    c = torch.randn((batch, m, n), device="cuda", generator=g)
    add = torch.randn((batch, m, n), device="cuda", generator=g) if terms in ("addend", "all") else None
    bias = torch.randn(n, device="cuda", generator=g) if terms in ("bias", "all") else None
    beta = -0.5 if terms in ("beta", "all") else 0.0
    want = 0.75 * (a.double() @ b.double().transpose(1, 2)) + beta * c.double()
    size = 0.75 * (a.double().abs() @ b.double().abs().transpose(1, 2))
    want = want + (0 if add is None else add.double()) + (0 if bias is None else bias.double())
    want = want.relu() if act == ACT_RELU else want.sigmoid() if act == ACT_SIGMOID else want
    want = torch.softmax(want, -1)
    device.gemm(a, b, c, m=m, n=n, k=k, batch=batch, trans_b=True, stride_a=m * k, stride_b=n * k, stride_c=m * n,
                alpha=0.75, beta=beta, addend=add, stride_addend=m * n if add is not None else 0, bias=bias,
                activation=act, math=MATH_TF32, io_flags=IO_SOFTMAX)
    assert not device.gemm_timed_out()
    err = 2.0 ** -8 * float(size.max()) + 1e-5
    assert ((c - want).abs() <= err * want).all()
