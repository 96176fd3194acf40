"""The vector NTT pass at the edges of its shapes: transforms shorter than a
block's 4096 elements, one and several passes, columns and tables at addresses
that rule 16-byte accesses out, columns behind a device pointer array."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from vortexstark_b200 import ntt
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
