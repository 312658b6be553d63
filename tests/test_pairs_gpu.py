"""The two-paths-per-thread kernels against the one-path kernels.

A pass over P paths must not depend on how it is split into batches.  Small
batches run one path per thread and a single tile of variates per CTA, large
ones two paths per thread with the last rates in tensor memory and several
tiles per CTA; both evaluate the same sequence of roundings per path, so the
results are compared bit for bit.
"""
from __future__ import annotations

import ctypes
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BATCH = 16384  # one path per thread


def pipeline(model, n, F, **kw):
    from useful_code_b200 import market as mk
    from useful_code_b200.pricer import Pipeline

    cfg = mk.make_config(model)
    f0 = np.resize(cfg.f0, n).astype(np.float32)
    return Pipeline(mk.build_market(replace(cfg, n=n, F=F, f0=f0, **kw)))


# rates around the multiples of four and the shared / tensor memory split,
# every compiled factor count and the generic one, odd path counts
SHAPES = [("c3", 80, 10, 100003), ("c2", 40, 5, 160001), ("c5", 120, 15, 100511),
          ("c2", 37, 5, 163333), ("c3", 128, 10, 100481), ("c5", 61, 16, 100737),
          ("c3", 50, 4, 165601), ("c2", 47, 3, 160961), ("c3", 19, 16, 104001)]


@pytest.mark.parametrize("model,n,F,P", SHAPES)
def test_first_pass_batches(cuda, model, n, F, P):
    pipe = pipeline(model, n, F)
    whole = pipe.first_pass(P, 777)
    parts = pipe.first_pass(P, 777, batch=BATCH)
    for name in ("vars", "ex", "cf", "num"):
        assert torch.equal(getattr(whole, name), getattr(parts, name)), name


@pytest.mark.parametrize("model,n,F,P", SHAPES)
@pytest.mark.parametrize("product", ["swaption", "cancellable", "bermudan_cap"])
def test_second_pass_batches(cuda, model, n, F, P, product):
    pipe = pipeline(model, n, F, product=product)
    rule = pipe.regress(pipe.first_pass(8192, 0))
    whole = pipe.second_pass(P, 99999, rule)
    parts = pipe.second_pass(P, 99999, rule, batch=BATCH)
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("product", ["european", "tarn"])
@pytest.mark.parametrize("n,F,P", [(20, 3, 150001), (49, 10, 60000)])
def test_strip_batches(cuda, n, F, P, product):
    pipe = pipeline("c1" if product == "european" else "t1", n, F, product=product)
    whole = pipe.second_pass(P, 5, None)
    assert torch.equal(whole, pipe.second_pass(P, 5, None, batch=BATCH))


def test_nested_rule_batches(cuda):
    from useful_code_b200.pricer import Selector

    pipe = pipeline("c3", 44, 10)
    rule = pipe.regress_nested(pipe.first_pass(1 << 14, 0), Selector.production(3))
    whole = pipe.second_pass(100001, 1 << 20, rule)
    assert torch.equal(whole, pipe.second_pass(100001, 1 << 20, rule, batch=BATCH))


@pytest.mark.parametrize("n,F,P,offset", [(80, 10, 300001, 123456), (20, 16, 400000, 127),
                                          (128, 3, 500002, 0), (2, 1, 700, 128)])
def test_variates_pieces(cuda, n, F, P, offset):
    """Several tiles per CTA (large P) against single tiles at other offsets
    of the tile grid."""
    from useful_code_b200._lib import call
    from useful_code_b200.pricer import dp, stream_handle

    pipe = pipeline("c3", n, F)
    addr = ctypes.addressof(pipe.model)
    whole = torch.empty(n, F, P, device="cuda")
    call("lmm_fused_variates", addr, P, offset, dp(whole), stream_handle())
    for lo, size in ((0, 301), (301, 350), (P // 2, 257), (P - 129, 129)):
        piece = torch.empty(n, F, size, device="cuda")
        call("lmm_fused_variates", addr, size, offset + lo, dp(piece), stream_handle())
        assert torch.equal(whole[:, :, lo:lo + size], piece), lo
