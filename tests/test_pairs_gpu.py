"""The two-paths-per-thread kernels against the one-path kernels.

A pass over P paths must not depend on how it is split into batches.  Small
batches run one path per thread and a single tile of variates per CTA, large
ones two paths per thread with the last rates in tensor memory and several
tiles per CTA; both evaluate the same sequence of roundings per path, so the
results are compared bit for bit.
"""
from __future__ import annotations

import ctypes
import threading
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
          ("c3", 50, 4, 165601), ("c2", 47, 3, 160961), ("c3", 19, 16, 104001),
          ("c2", 64, 3, 160233), ("c2", 57, 5, 161003), ("c5", 70, 16, 100111)]


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


@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 8, 9, 16, 31, 33, 63, 64, 65, 100, 127, 128])
def test_variates_depth_first_bridge(cuda, n):
    """Every tree shape of the depth-first bridge (the first of 100,000 paths) and
    of the level-by-level one (300 paths alone) against the construction in FP64
    on exact normals.  Bridge values reach 6 sqrt(128) =
    68; an FP32 combination rounds them by up to 68 * 2^-23 = 8e-6 per level
    (at most eight levels) and the rational inverse normal is within 7e-7
    relative of the exact one: 1e-4 bounds the difference of two points."""
    from scipy.special import ndtri

    from useful_code_b200 import market as mk
    from useful_code_b200._lib import call
    from useful_code_b200.pricer import LmmModel, LmmProduct, dp, stream_handle  # noqa: F401

    F, P, offset = 2, 300, 1000
    pipe = pipeline("c3", n, F)
    n_, alloc = n, np.zeros(F * n, np.int32)
    model = pipe.model
    taus = np.full(n_, 0.25, np.float32)
    disp = np.full(n_, 0.015, np.float32)
    f0 = np.full(n_, 0.04, np.float32)
    dirs = mk.sobol_directions(F * n_)
    scr = mk.scramblers(7, F * n_)
    d_dirs = torch.from_numpy(dirs.astype(np.int32)).cuda()
    d_scr = torch.from_numpy(scr.astype(np.int32)).cuda()
    vp = ctypes.c_void_p
    m = LmmModel(n_, F, vp(taus.ctypes.data), vp(disp.ctypes.data), vp(f0.ctypes.data),
                 model.d_A, model.d_fixed_drifts, dp(d_dirs), dp(d_scr), F * n_, 10.0)
    out = torch.empty(n_, F, P, device="cuda")
    call("lmm_fused_variates", ctypes.addressof(m), P, offset, dp(out), stream_handle())
    many = torch.empty(n_, F, 100000, device="cuda")
    call("lmm_fused_variates", ctypes.addressof(m), 100000, offset, dp(many), stream_handle())
    assert torch.equal(many[:, :, :P], out)
    lw, rw, sd = (np.zeros(n_) for _ in range(3))
    left, right, bidx = (np.zeros(n_, np.int32) for _ in range(3))
    call("lmm_bridge_tables_host", n_, *(vp(a.ctypes.data)
                                         for a in (lw, rw, sd, left, right, bidx)))
    call("lmm_bridge_allocate_diagonal", F, n_, vp(alloc.ctypes.data))
    idx = np.arange(1 + offset, 1 + offset + P, dtype=np.uint64)
    gray = idx ^ (idx >> np.uint64(1))
    ref = np.zeros((n_, F, P))
    for f in range(F):
        W = np.zeros((n_, P))
        for i in range(n_):
            d = alloc.reshape(F, n_)[f, i]
            x = np.full(P, scr[d], np.uint32)
            for b in range(12):
                x ^= np.where((gray >> np.uint64(b)) & np.uint64(1), dirs[d, b], 0).astype(
                    np.uint32)
            z = ndtri(np.clip(x.astype(np.float64), 1.0, None) * 2.0 ** -32)
            y = sd[i] * z
            if i > 0:
                y += rw[i] * W[right[i]]
                if left[i] > 0:
                    y += lw[i] * W[left[i] - 1]
            W[bidx[i]] = y
        ref[:, f] = np.diff(W, axis=0, prepend=0.0)
    assert np.max(np.abs(out.cpu().numpy() - ref)) < 1e-4


def test_tensor_memory_handed_over(cuda):
    """CTAs of two launches on two streams share the SMs and take over one
    another's tensor-memory columns (a few hundred CTAs each, three per SM):
    every pass gives the bits it gives alone."""
    pipes = [pipeline("c3", 80, 10), pipeline("c3", 80, 10)]
    rule = pipes[0].regress(pipes[0].first_pass(8192, 0))
    P = 150001
    alone = pipes[0].second_pass(P, 4242, rule)
    first = pipes[1].first_pass(P, 4242)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(4):
        with torch.cuda.stream(streams[0]):
            pay = pipes[0].second_pass(P, 4242, rule)
        with torch.cuda.stream(streams[1]):
            ls = pipes[1].first_pass(P, 4242)
        torch.cuda.synchronize()
        assert torch.equal(pay, alone)
        assert torch.equal(ls.vars, first.vars) and torch.equal(ls.num, first.num)


def test_threads_price_at_once(cuda):
    """Two host threads launch the same kernels with different amounts of
    shared memory (the segments of a chain, models of other sizes): neither
    takes away the other's, and each gets the payoffs it gets alone."""
    P = 100003
    pipes = [pipeline("c3", 80, 10), pipeline("c3", 128, 10)]
    rules = [p.regress(p.first_pass(8192, 0)) for p in pipes]
    alone = [p.second_pass(P, 4242, r) for p, r in zip(pipes, rules)]
    torch.cuda.synchronize()
    errors = []

    def price(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(40):
                    pay = pipes[k].second_pass(P, 4242, rules[k])
                if not torch.equal(pay, alone[k]):
                    errors.append(f"thread {k}: other payoffs")
        except RuntimeError as e:
            errors.append(f"thread {k}: {e}")

    threads = [threading.Thread(target=price, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


# the reverse sweep takes two paths per thread from 75,777 paths (593 tiles, up
# to 10 factors), the recompute and a recording pass in one launch from 56,833
# (n F P >= 2^23), a recording pass in segments as test_chain_batches; 15 factors
# and the generic form keep one in the reverse sweep
@pytest.mark.parametrize("model,n,F,P,product", [
    ("c3", 80, 10, 110004, "swaption"), ("c2", 40, 5, 81932, "cancellable"),
    ("c2", 40, 5, 250020, "swaption"), ("c5", 120, 15, 150004, "cancellable"),
    ("c2", 64, 3, 262148, "swaption"),
    ("c3", 24, 10, 77828, "bermudan_cap"), ("c1", 28, 5, 75780, "european"),
    ("c2", 37, 3, 82052, "swaption"), ("c5", 30, 15, 60004, "swaption"),
    ("c3", 21, 16, 57004, "cancellable")])
def test_greeks_batches(cuda, model, n, F, P, product):
    """Greeks of P paths are the path-weighted sums of its batches' Greeks.
    Per path every value is the same; a thread's and a warp's FP32 sums join
    64 paths of the batch's instead of 32, and each of the up to 63 additions
    rounds its partial sum by 2^-24 at most.  Rows of dV/dA cancel little, so
    the 2-norm differs by less than 63 * 2^-24 = 3.8e-6 of the result."""
    pipe = pipeline(model, n, F, product=product)
    euro = product == "european"
    rule = None if euro else pipe.regress(pipe.first_pass(8192, 0))
    whole = pipe.greeks(P, 99999, rule)
    price, delta, abar, vega, ex = 0.0, 0.0, 0.0, 0.0, []
    for lo in range(0, P, BATCH):
        size = min(BATCH, P - lo)
        g = pipe.greeks(size, 99999 + lo, rule)
        w = size / P
        price += w * g.price
        delta, abar, vega = delta + w * g.delta, abar + w * g.abar, vega + w * g.vega_rate
        ex.append(g.exercise_step)
    assert np.array_equal(whole.exercise_step, np.concatenate(ex))
    assert abs(whole.price - price) < 1e-12 * abs(price)
    for name, ref in (("delta", delta), ("abar", abar), ("vega_rate", vega)):
        got = getattr(whole, name)
        assert np.linalg.norm(got - ref) < 3.8e-6 * np.linalg.norm(ref), name


@pytest.mark.parametrize("model,n,F,K", [("c3", 16, 10, 57007), ("c2", 30, 5, 57004),
                                         ("c3", 50, 3, 57001), ("c5", 28, 15, 20485),
                                         ("c3", 27, 16, 20483)])
def test_bound_outer_paths(cuda, model, n, F, K):
    """Outer paths of the Andersen-Broadie bound, two per thread, against a
    call with fewer, one per thread: states, decisions, exercise values and the
    continuation estimates from them (inner paths are counted by the outer
    path's number), bit for bit."""
    pipe = pipeline(model, n, F, product="swaption")
    rule = pipe.regress(pipe.first_pass(8192, 0))
    whole = pipe.andersen_broadie(rule, K, 4321, 128, keep=True)
    few = 501
    part = pipe.andersen_broadie(rule, few, 4321, 128, keep=True)
    for name in ("ckpt", "ckptN", "X", "Z", "Q"):
        assert torch.equal(getattr(whole, name)[..., :few], getattr(part, name)), name
    tail = pipe.andersen_broadie(rule, 257, 4321 + K - 257, 128, keep=True)
    for name in ("ckpt", "ckptN", "X", "Z"):
        assert torch.equal(getattr(whole, name)[..., K - 257:], getattr(tail, name)), name


@pytest.mark.parametrize("n,F", [(2, 1), (2, 2), (16, 4), (20, 3), (40, 5), (80, 10),
                                 (128, 16)])
@pytest.mark.parametrize("P,offset", [(1, 0), (127, 126), (129, 127), (4099, 2**31 - 4102)])
def test_variates_by_level(cuda, n, F, P, offset):
    """Few paths (level by level, tiles of 128) against the same paths inside a
    launch with many (depth first; one factor stays level by level up to 94,720
    paths); the last offset ends at the last index."""
    from useful_code_b200._lib import call
    from useful_code_b200.pricer import dp, stream_handle

    pipe = pipeline("c3", n, F)
    few = torch.empty(n, F, P, device="cuda")
    call("lmm_fused_variates", ctypes.addressof(pipe.model), P, offset, dp(few), stream_handle())
    before = 100000 if offset > 200000 else 0
    size = before + P if before else 100000
    many = torch.empty(n, F, size, device="cuda")
    call("lmm_fused_variates", ctypes.addressof(pipe.model), size, offset - before, dp(many),
         stream_handle())
    assert torch.equal(few, many[:, :, before:before + P])


# chains of segments take two paths per thread later than one launch does
@pytest.mark.parametrize("model,n,F,P", [("c3", 80, 10, 110011), ("c2", 40, 5, 250017),
                                         ("c5", 120, 15, 150011), ("c2", 64, 3, 262147),
                                         ("c3", 128, 10, 100481)])
@pytest.mark.parametrize("product", ["swaption", "cancellable"])
def test_chain_batches(cuda, model, n, F, P, product):
    """A chain with two paths per thread against batches with one."""
    pipe = pipeline(model, n, F, product=product)
    rule = pipe.regress(pipe.first_pass(8192, 0))
    whole = pipe.second_pass(P, 99999, rule)
    assert torch.equal(whole, pipe.second_pass(P, 99999, rule, batch=BATCH))


@pytest.mark.parametrize("model,n,F", [("c3", 128, 10), ("c5", 120, 15), ("c2", 12, 2),
                                       ("c2", 20, 3), ("c2", 14, 5), ("c3", 20, 10)])
@pytest.mark.parametrize("product", ["swaption", "bermudan_cap"])
def test_more_ctas_than_fit(cuda, model, n, F, product):
    """One path per thread with more CTAs than the form that loads a step ahead
    has places for (it reads rows and normals at the step then) against small
    batches, which load ahead."""
    pipe = pipeline(model, n, F, product=product)
    P = 95001 if n * F <= 200 else 40001
    whole, parts = pipe.first_pass(P, 777), pipe.first_pass(P, 777, batch=BATCH)
    for name in ("vars", "ex", "cf", "num"):
        assert torch.equal(getattr(whole, name), getattr(parts, name)), name
    rule = pipe.regress(parts)
    assert torch.equal(pipe.second_pass(P, 99999, rule),
                       pipe.second_pass(P, 99999, rule, batch=BATCH))
