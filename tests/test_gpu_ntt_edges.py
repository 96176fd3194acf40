"""The vector NTT pass at the edges of its shapes: transforms shorter than a
block's 4096 elements, one and several passes, columns and tables at addresses
that rule 16-byte accesses out, columns behind a device pointer array."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from vortexstark_b200 import ntt, tune
from vortexstark_b200.circle import Coset
from vortexstark_b200.workload import m31_array

pytestmark = pytest.mark.gpu


def _shifted(words, by):
    """The same words `by` words past a 16-byte boundary."""
    import torch
    t = torch.zeros(len(words) + by + 4, dtype=torch.int32, device="cuda")
    v = t[by:by + len(words)]
    v.copy_(to_dev(words))
    return v


@pytest.mark.parametrize("log_n", list(range(4, 18)) + [19, 21])
@pytest.mark.parametrize("by", [0, 1, 2])
def test_natural_order(oracle, log_n, by):
    coset = Coset.half_coset(log_n)
    oc = oracle.coset("half_coset", log_n)
    cache = ntt.TwiddleCache(coset)
    x = m31_array(50 + log_n, 1 << log_n)
    ev = oracle.ntt_evaluate(x, oc)
    tables = ("d_twiddles", "d_circle_twids", "d_itwiddles", "d_circle_itwids")
    for shift_tables in (0, 1) if by else (0,):
        if shift_tables:
            for name in tables:
                setattr(cache, name, _shifted(to_host(getattr(cache, name)), by))
        d = _shifted(x, by)
        ntt.evaluate(d, cache)
        assert np.array_equal(to_host(d), ev)
        ntt.interpolate(d, cache)
        assert np.array_equal(to_host(d), x)


@pytest.mark.parametrize("log_n", [5, 8, 11, 12, 13, 16, 18])
def test_columns_of_mixed_alignment(oracle, log_n):
    cols = [m31_array(90 + c, 1 << log_n) for c in range(3)]
    oc = oracle.coset("half_coset", log_n)
    cache = ntt.TwiddleCache(Coset.half_coset(log_n))
    d = [_shifted(c, by) for c, by in zip(cols, (0, 1, 4))]
    ntt.evaluate_batch(d, cache)
    for c, t in zip(cols, d):
        assert np.array_equal(to_host(t), oracle.ntt_evaluate(c, oc))
    ntt.interpolate_batch(d, cache)
    for c, t in zip(cols, d):
        assert np.array_equal(to_host(t), c)
    stw = ntt.StwoNttCache(log_n)
    ntt.evaluate_stwo_batch(d, stw)
    for c, t in zip(cols, d):
        assert np.array_equal(to_host(t), oracle.stwo_ntt_evaluate(c))
    ntt.interpolate_stwo_batch(d, stw)
    for c, t in zip(cols, d):
        assert np.array_equal(to_host(t), c)


def _repacked(cache, gap):
    """The line tables with `gap` unused words ahead of every layer."""
    offs = [o + (i + 1) * gap for i, o in enumerate(cache.layer_offsets)]
    for name in ("d_twiddles", "d_itwiddles"):
        old = to_host(getattr(cache, name))
        new = np.full(len(old) + gap * len(offs), 0x7FFFFFFE, dtype=np.uint32)
        for o, p, n in zip(cache.layer_offsets, offs, cache.layer_sizes):
            new[p:p + n] = old[o:o + n]
        setattr(cache, name, to_dev(new))
    cache.layer_offsets = offs


@pytest.mark.parametrize("gap", [1, 2, 3, 4])
@pytest.mark.parametrize("log_n", [4, 5, 8, 10, 12, 14, 17, 21, 22])
def test_layer_offsets_of_the_caller(oracle, log_n, gap):
    """Layers at word offsets that no wide load may start at."""
    coset = Coset.half_coset(log_n)
    oc = oracle.coset("half_coset", log_n)
    cache = ntt.TwiddleCache(coset)
    _repacked(cache, gap)
    cols = [m31_array(70 + log_n + c, 1 << log_n) for c in range(2)]
    evs = [oracle.ntt_evaluate(c, oc) for c in cols]
    d = [to_dev(c) for c in cols]
    ntt.evaluate(d[0], cache)
    assert np.array_equal(to_host(d[0]), evs[0])
    ntt.interpolate(d[0], cache)
    ntt.evaluate_batch(d, cache)
    assert all(np.array_equal(to_host(x), e) for x, e in zip(d, evs))
    ntt.interpolate_batch(d, cache)
    assert all(np.array_equal(to_host(x), c) for x, c in zip(d, cols))


TABLES = ("d_twiddles", "d_circle_twids", "d_itwiddles", "d_circle_itwids")


def _shift_tables(cache, names, by):
    for name in names:
        setattr(cache, name, _shifted(to_host(getattr(cache, name)), by))


@pytest.mark.parametrize("tables", [False, True])
@pytest.mark.parametrize("log_n,by", [(18, 1), (20, 3), (22, 1), (22, 2)])
def test_unaligned_long_columns(oracle, log_n, by, tables):
    """2^20 and 2^22 elements in one column: the vector pass with twiddles up
    front and, above four blocks per SM, without."""
    coset = Coset.half_coset(log_n)
    cache = ntt.TwiddleCache(coset)
    if tables:
        _shift_tables(cache, TABLES, by)
    x = m31_array(150 + log_n, 1 << log_n)
    d = _shifted(x, by)
    ntt.evaluate(d, cache)
    assert np.array_equal(to_host(d), oracle.ntt_evaluate(x, oracle.coset("half_coset", log_n)))
    ntt.interpolate(d, cache)
    assert np.array_equal(to_host(d), x)


@pytest.mark.parametrize("n_cols,log_n", [(3, 5), (3, 8), (3, 11), (3, 12), (3, 13), (3, 16), (16, 18)])
@pytest.mark.parametrize("by", [1, 2, 3])
def test_columns_with_unaligned_tables(oracle, n_cols, log_n, by):
    cols = [m31_array(190 + c, 1 << log_n) for c in range(n_cols)]
    oc = oracle.coset("half_coset", log_n)
    cache = ntt.TwiddleCache(Coset.half_coset(log_n))
    _shift_tables(cache, TABLES, by)
    d = [_shifted(c, (by + i) % 4) for i, c in enumerate(cols)]
    ntt.evaluate_batch(d, cache)
    for x, c in zip(d[:3], cols):
        assert np.array_equal(to_host(x), oracle.ntt_evaluate(c, oc))
    ntt.interpolate_batch(d, cache)
    assert all(np.array_equal(to_host(x), c) for x, c in zip(d, cols))
    plain, stwo = ntt.StwoNttCache(log_n), ntt.StwoNttCache(log_n)
    _shift_tables(stwo, ("d_fwd_twiddles", "d_inv_twiddles"), by)
    want = [to_dev(c) for c in cols]
    ntt.evaluate_stwo_batch(want, plain)
    ntt.evaluate_stwo_batch(d, stwo)
    assert all(np.array_equal(to_host(x), to_host(w)) for x, w in zip(d, want))
    ntt.interpolate_stwo_batch(d, stwo)
    assert all(np.array_equal(to_host(x), c) for x, c in zip(d, cols))


@pytest.mark.parametrize("gap", [0, 1])
@pytest.mark.parametrize("upper", range(3, 10))
def test_every_upper_shape_with_unaligned_tables(oracle, upper, gap):
    """A bottom pass of 12 layers and one upper pass of `upper`, on tables one
    word off and on layers one word off."""
    log_n = 12 + upper
    tune.set_ntt_plan(log_n, 12, upper)
    try:
        cache = ntt.TwiddleCache(Coset.half_coset(log_n))
        if gap:
            _repacked(cache, gap)
        else:
            _shift_tables(cache, TABLES, 1)
        cols = [m31_array(230 + upper + c, 1 << log_n) for c in range(2)]
        d = [_shifted(c, 2 * i) for i, c in enumerate(cols)]
        ntt.evaluate_batch(d, cache)
        oc = oracle.coset("half_coset", log_n)
        assert all(np.array_equal(to_host(x), oracle.ntt_evaluate(c, oc)) for x, c in zip(d, cols))
        ntt.interpolate_batch(d, cache)
        assert all(np.array_equal(to_host(x), c) for x, c in zip(d, cols))
    finally:
        tune.set_ntt_plan(log_n, 0, 0)
