"""The kernels' own divisions on the device against `/` and against the host's
IEEE quotient, bit for bit: the restart path's guarded division (div1 in
opencaeporo_b200/csrc/flash_div.cuh) for every kind of operand, its unguarded
one (div_core) for those it admits, the division by a constant (div_const in
flash_common.cuh) on both sides of its window of 2^-896 .. 2^896, and the error
of the reciprocal that div_core starts from, which tests/test_div_core.py
takes to be below 2^-19."""
import numpy as np
import pytest

D1, D2 = 2.41421356237, -0.41421356237


def _run(form, a, b):
    import torch
    from opencaeporo_b200 import _lib
    x, y = torch.as_tensor(a).cuda(), torch.as_tensor(b).cuda()
    q = torch.empty_like(x)
    _lib.check(_lib.lib().ocpf_check_division(form, x.numel(), x.data_ptr(), y.data_ptr(), q.data_ptr(), None),
               "ocpf_check_division")
    torch.cuda.synchronize()
    return q.cpu().numpy()


def _mantissas(rng, n):
    """Random ones, with runs of zeros and of ones among them."""
    m = rng.integers(0, 1 << 52, n)
    m[: n // 16] &= rng.integers(0, 1 << 52, n // 16) & rng.integers(0, 1 << 52, n // 16)
    m[n // 16: n // 8] |= ((1 << 52) - 1) ^ rng.integers(0, 16, n // 8 - n // 16)
    m[n // 8: 3 * n // 16] = rng.integers(0, 16, 3 * n // 16 - n // 8)
    return m


def _numbers(rng, n, lo, hi):
    """Magnitudes of 2^lo .. 2^(hi + 1), random signs."""
    e = rng.integers(lo, hi + 1, n) + 1023
    bits = (e.astype(np.uint64) << np.uint64(52)) | _mantissas(rng, n).astype(np.uint64)
    return bits.view(np.float64) * np.where(rng.integers(0, 2, n) > 0, 1.0, -1.0)


def _special():
    ones = float(2 ** 53 - 1)
    v = [0.0, np.inf, np.nan, 5e-324, 2.0 ** -1030, 2.0 ** -1022, np.finfo(float).max, 1.0, 3.0, ones, ones * 2.0 ** -53,
         ones * 2.0 ** 300, ones * 2.0 ** -300]
    for k in (-897, -896, -451, -450, -449, 449, 450, 451, 895, 896, 897):
        v += [2.0 ** k, np.nextafter(2.0 ** k, 0), np.nextafter(2.0 ** k, np.inf)]
    v = np.array(v)
    return np.concatenate([v, -v])


def _same(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.int64), want[ok].view(np.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("span", [8, 449, 1000])
def test_guarded_division_is_the_quotient(span):
    rng = np.random.default_rng(span)
    a, b = _numbers(rng, 1 << 20, -span, span), _numbers(rng, 1 << 20, -span, span)
    s = _special()
    a = np.concatenate([a, np.repeat(s, len(s)), a[:4096], np.resize(s, 4096)])
    b = np.concatenate([b, np.tile(s, len(s)), np.resize(s, 4096), b[:4096]])
    with np.errstate(all="ignore"):
        want = a / b
    _same(_run(0, a, b), want)
    _same(_run(1, a, b), want)


@pytest.mark.gpu
@pytest.mark.parametrize("span", [8, 449])
def test_unguarded_division_is_the_quotient_for_what_it_admits(span):
    rng = np.random.default_rng(100 + span)
    a, b = _numbers(rng, 1 << 20, -span, span), _numbers(rng, 1 << 20, -span, span)
    ones = (b.view(np.int64) & ((1 << 52) - 1)) == (1 << 52) - 1
    assert ones.any()
    a, b = a[~ones], b[~ones]
    _same(_run(2, a, b), a / b)


@pytest.mark.gpu
@pytest.mark.parametrize("form,d", [(3, 3.0), (4, 9.0), (5, 54.0), (6, D1 - D2)])
def test_division_by_a_constant_is_the_quotient(form, d):
    rng = np.random.default_rng(form)
    a = np.concatenate([_numbers(rng, 1 << 20, -1000, 1000), _numbers(rng, 1 << 16, -898, -894),
                        _numbers(rng, 1 << 16, 894, 898), _special()])
    with np.errstate(all="ignore"):
        want = a / d
    _same(_run(form, a, np.full_like(a, d)), want)


@pytest.mark.gpu
def test_error_of_the_start():
    rng = np.random.default_rng(7)
    m = np.concatenate([_mantissas(rng, 1 << 22), np.arange(1 << 20) << 32])
    b = ((np.uint64(1023) << np.uint64(52)) | m.astype(np.uint64)).view(np.float64)
    e = _run(7, b, b * 2.0 ** rng.integers(-449, 450, len(b)))
    assert np.abs(e).max() < 2.0 ** -19


def test_check_division_rejects_bad_arguments():
    from opencaeporo_b200 import _lib
    f = _lib.lib().ocpf_check_division
    assert f(8, 1, None, None, None, None) != 0
    assert f(-1, 0, None, None, None, None) != 0
    assert f(1, -1, None, None, None, None) != 0
    assert f(1, 4, None, None, None, None) != 0
    assert f(1, 0, None, None, None, None) == 0
