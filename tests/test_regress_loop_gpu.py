"""The one-launch backward regression loop against one launch per date, in
graphs, on part of the GPU and on two streams."""
from __future__ import annotations

import threading
from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu


# drop: every date's last basis functions left out, so that no date has a
# table the kernels know
@pytest.mark.parametrize("model,P,drop", [("c2", 1, 0), ("c2", 31, 0), ("c2", 4099, 0),
                                          ("c3", 513, 0), ("c3", 60001, 0), ("c3", 8192, 1),
                                          ("c2", 5001, 1), ("c5", 2049, 0), ("c5", 50003, 0)])
@pytest.mark.parametrize("normalise", [True, False])
def test_regression_loop_equals_dates(cuda, model, P, drop, normalise):
    """The one-launch backward loop against one launch per date (the sharded
    protocol with one shard): the same sums in the same order."""
    from useful_code_b200 import market as mk
    from useful_code_b200.pricer import Pipeline
    from useful_code_b200.sharded import regress_sharded

    cfg = mk.make_config(model)
    pipe = Pipeline(mk.build_market(replace(cfg, normalise=normalise)))
    pipe._nbasis[:] = (pipe._nbasis - drop).clip(1)
    ls = pipe.first_pass(P, 31)
    one = pipe.regress(ls)
    dates = regress_sharded(pipe, ls, P)
    # the dates divide their sums by the paths in another kernel: the same
    # FP64 operations, so equal bits
    assert torch.equal(one.beta, dates.beta)
    assert int(one.status) == int(dates.status)
    assert abs(float(one.price) - float(dates.price)) <= 1e-12 * abs(float(dates.price))


def c3_pipeline():
    from useful_code_b200 import market as mk
    from useful_code_b200.pricer import Pipeline

    return Pipeline(mk.build_market(mk.make_config("c3")))


def test_regression_graph(cuda):
    """The loop captured as a CUDA graph: each replay regresses what the
    inputs hold then."""
    pipe = c3_pipeline()
    P = 30001
    ls, other = pipe.first_pass(P, 31), pipe.first_pass(P, 90000)
    pipe.regress(ls)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = pipe.regress(ls)
    for inputs in (ls, other):
        for name in ("vars", "ex", "cf", "num"):
            getattr(ls, name).copy_(getattr(inputs, name))
        graph.replay()
        torch.cuda.synchronize()
        direct = pipe.regress(ls)
        assert torch.equal(out.beta, direct.beta) and torch.equal(out.price, direct.price)


@pytest.fixture
def sixteen_sms(cuda):
    """A stream of a green context with 16 of the GPU's SMs."""
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r
        return r[1:] if len(r) > 2 else r[1] if len(r) == 2 else None

    kind = cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM
    device = ok(cu.cuDeviceGet(0))
    groups, _, _ = ok(cu.cuDevSmResourceSplitByCount(1, ok(cu.cuDeviceGetDevResource(device, kind)),
                                                     0, 16))
    green = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc([groups[0]], 1)), device,
                                   cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(stream))
    torch.cuda.synchronize()
    ok(cu.cuStreamDestroy(stream))
    ok(cu.cuGreenCtxDestroy(green))


@pytest.mark.parametrize("P", [4099, 60001])
def test_regressions_on_part_of_the_gpu(sixteen_sms, P):
    """On a stream that owns 16 SMs no cooperative launch of more CTAs fits:
    the regression runs date by date, with the same bits; the nested one with
    16 CTAs, whose FP64 sums over CTAs round differently (2^-53 per term of
    sums that the coefficients amplify by the Grams' condition, below 1e6)."""
    from useful_code_b200.pricer import Selector

    pipe = c3_pipeline()
    ls = pipe.first_pass(P, 31)
    whole, nested = pipe.regress(ls), pipe.regress_nested(ls, Selector.production(3, 300))
    torch.cuda.synchronize()
    with torch.cuda.stream(sixteen_sms):
        part, part_nested = pipe.regress(ls), pipe.regress_nested(ls, Selector.production(3, 300))
    torch.cuda.synchronize()
    assert torch.equal(whole.beta, part.beta) and torch.equal(whole.price, part.price)
    assert int(part.status) == int(whole.status)
    assert int(part_nested.status) == int(nested.status)
    assert torch.equal(part_nested.npaths, nested.npaths)
    scale = nested.beta.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)
    assert float(((part_nested.beta - nested.beta).abs() / scale).max()) < 1e-9


def test_regressions_on_two_streams(cuda):
    """Two threads regress at once, each launch wanting every SM for itself:
    they take turns and give the bits they give alone."""
    from useful_code_b200.pricer import Selector

    pipes = [c3_pipeline(), c3_pipeline()]
    inputs = [p.first_pass(60001, 31 + 70000 * k) for k, p in enumerate(pipes)]
    sel = Selector.production(3, 300)
    alone = [(p.regress(x), p.regress_nested(x, sel)) for p, x in zip(pipes, inputs)]
    torch.cuda.synchronize()
    errors = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                got = pipes[k].regress(inputs[k]), pipes[k].regress_nested(inputs[k], sel)
                for a, b in zip(got, alone[k]):
                    if int(a.status) != int(b.status) or not torch.equal(a.beta, b.beta):
                        errors.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
