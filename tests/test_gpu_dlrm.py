"""End-to-end parity of the DLRM-style step with the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

import torch
import annc_b200  # noqa: F401,E402  (no fallback: a missing library fails the collection)
from annc_b200 import synth  # noqa: E402
from annc_b200._lib import MATH_AUTO, MATH_FP32  # noqa: E402
from annc_b200.dlrm import DlrmPipeline  # noqa: E402


@pytest.mark.parametrize("math,tol", [(MATH_FP32, 2e-5), (MATH_AUTO, 2e-3)])
def test_dlrm_step_matches_oracle(math, tol):
    model = synth.dlrm_model(seed=3, batch=4096, max_rows=3e5)
    pipe = DlrmPipeline(model, torch.device("cuda:0"), math=math, keep_host_inputs=True)
    got = pipe.forward().cpu().numpy()
    assert pipe.embed_error_bits() == 0
    want = oracle.dlrm_forward(model, threads=oracle.host_threads())
    assert np.abs(got - want).max() <= tol  # sigmoid outputs in (0,1): absolute == normwise
    # the end-to-end entry (host buffers in, host result out) gives the same answer
    pipe.ids_all.zero_()
    pipe.seg_all.zero_()
    pipe.dense.zero_()
    h = pipe.forward_e2e()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(h.numpy(), got)


def test_pipelined_steps_of_another_stream_are_waited_for():
    """Steps issued under one stream, sync_pipeline() and the reads on another: the results are
    complete there, and a forward() after it does not write over a buffer set still in use."""
    model = synth.dlrm_model(seed=4, batch=8192, max_rows=2e4)
    pipe = DlrmPipeline(model, torch.device("cuda:0"))
    want = pipe.forward().clone()
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    for steps in (1, 2, 3):
        for b in pipe._bufs:
            b["acts_t"][-1].fill_(-1.0)
        other.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(other):
            outs = [pipe.forward_pipelined() for _ in range(steps)]
        pipe.sync_pipeline()
        got = [o.clone() for o in outs[-2:]]
        again = pipe.forward().clone()
        torch.cuda.synchronize()
        for o in got + [again]:
            assert torch.equal(o, want)


@pytest.mark.parametrize("batch,max_bag,one", [(1, 3, True), (64, 120, True), (64, 130, False), (512, 20, True), (513, 20, False),
                                               (512, 24, False)])
def test_small_steps_on_one_stream(batch, max_bag, one):
    """Steps at either side of the lines between one stream and two (batch, lookups, mean bag): the oracle's predictions,
    and the same ones whichever way the steps are issued."""
    model = synth.dlrm_model(seed=6, batch=batch, max_rows=3e4, max_bag=max_bag)
    pipe = DlrmPipeline(model, torch.device("cuda:0"), keep_host_inputs=True)
    assert pipe._one_stream() is one
    outs = [pipe.forward().clone() for _ in range(3)]
    torch.cuda.synchronize()
    if one:  # waits for nothing of another stream: it can be captured as it is
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = pipe.forward()
        pipe.out.fill_(-1.0)
        graph.replay()
        outs.append(captured.clone())
    outs += [pipe.forward_pipelined() for _ in range(4)][2:]
    pipe.sync_pipeline()
    outs = [o.clone() for o in outs]
    outs.append(pipe.forward().clone())
    for _ in range(3):  # from host inputs
        for st in pipe.sets:
            st["ids_all"].zero_()
        torch.cuda.synchronize()
        pipe._prefetched = [False, False]
        host = pipe.forward_e2e()
        torch.cuda.synchronize()
        outs.append(host.cuda())
    assert pipe.embed_error_bits() == 0
    for o in outs:
        assert torch.equal(o, outs[0])
    want = oracle.dlrm_forward(model, threads=oracle.host_threads())
    assert np.abs(outs[0].cpu().numpy() - want).max() <= 2e-3


def test_smoke_entry():
    import __graft_entry__ as g
    g.smoke()
