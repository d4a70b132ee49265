"""Single device functions against their definition, where whole steps do not
reach every branch: the grouped FP64 reciprocals of the WENO weights against
the division operator, bit for bit, and the FP32 WENO interface values
against 64 bits."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUILD = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-x_b200", "_build")


def _lib(name):
    return ctypes.CDLL(os.path.join(BUILD, name))


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _bits(sign, exp, mant):
    u = (np.asarray(sign, np.uint64) << np.uint64(63)) | (np.asarray(exp, np.uint64) << np.uint64(52)) | \
        np.asarray(mant, np.uint64)
    return u.view(np.float64)


def _denominators():
    """Every exponent with random significands, and the values at which the
    branch-free sequence ends: 2^-400 and 2^400, significands of all ones,
    zeros, subnormals, infinities and NaN."""
    rng = np.random.default_rng(20261205)
    ones = (1 << 52) - 1
    exps = np.repeat(np.arange(0, 2048, dtype=np.uint64), 40)
    any_ = _bits(rng.integers(0, 2, exps.size), exps, rng.integers(0, ones + 1, exps.size))
    edge = [_bits(s, e, m) for s in (0, 1) for e in (0, 1, 2, 622, 623, 624, 1022, 1023, 1422, 1423, 1424, 2045, 2046)
            for m in (0, 1, 2, ones, ones - 1, ones - 2, ones - (1 << 20), (1 << 32) - 1, ones ^ 1, ones ^ (1 << 32),
                      ones ^ (1 << 51))]
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1.0, 1e-36])
    return np.concatenate([any_, np.array(edge).ravel(), special])


@pytest.mark.parametrize("group", [2, 3])
def test_grouped_reciprocals_equal_division(need_gpu, group):
    import torch
    lib = _lib("libfxb_test_exact.so")
    rng = np.random.default_rng(group)
    b = _denominators()
    plain = _bits(0, 1023 + rng.integers(-300, 300, b.size), rng.integers(0, 1 << 52, b.size))
    rows = [rng.permutation(b)[:b.size // group * group].reshape(-1, group)]     # any members together
    for q in range(group):                                                       # one member needs the division
        g = np.stack([rng.permutation(plain) for _ in range(group)], axis=1)
        g[:, q] = b
        rows.append(g)
    x = np.ascontiguousarray(np.concatenate(rows))
    d = torch.from_numpy(x).cuda()
    y = torch.empty_like(d)
    assert lib.fxt_recips(group, _p(d), _p(y), ctypes.c_long(len(x))) == 0
    got = y.cpu().numpy()
    with np.errstate(all="ignore"):
        want = 1.0 / x
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint64)[~nan], want.view(np.uint64)[~nan])


def _weno64(method, I):
    """(i + 1/2, i - 1/2) of stencils I[n][5], in 64 bits."""
    a, b, c, d, e = I.T
    p = [(2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6]
    m = [(-a + 5 * b + 2 * c) / 6, (2 * b + 5 * c - d) / 6, (11 * c - 7 * d + 2 * e) / 6]
    s = [13. / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
         13. / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
         13. / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2]
    out = []
    for g, v in (((0.1, 0.6, 0.3), p), ((0.3, 0.6, 0.1), m)):
        w = [g[q] * (1 + abs(s[0] - s[2]) / (1e-36 + s[q])) if method == 2 else g[q] / (1e-36 + s[q]) for q in range(3)]
        t = w[0] + w[1] + w[2]
        out.append(sum(w[q] * v[q] for q in range(3)) / t)
    return out


@pytest.mark.parametrize("method", [1, 2])
def test_mixed_weno_rounding(need_gpu, method):
    """Stencils of 1 + 0.1 noise; one ulp of 1 is u = 2^-23.  Largest error: the
    values are differences of at most 0.9 times coefficients that add up to 7/6
    at most, with the difference, the coefficient, the product and the sum
    rounded (4 u / 2 times 1.05), weights that are off by some 6 u / 2 times as
    much, and the last sum at the value's size (u / 2): 6 u.  Root mean square:
    0.23 u, the last sum and little else; 0.47 u where the candidates are formed
    at the value's size, 0.60 u and more where the weights' rounding multiplies
    them."""
    import torch
    lib = _lib("libfxb_test_mixed.so")
    rng = np.random.default_rng(7)
    n = 1 << 18
    x = (1.0 + 0.1 * rng.standard_normal((n, 5))).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    r, l = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    assert lib.fxt_weno_mixed(method, _p(d), _p(r), _p(l), ctypes.c_long(n)) == 0
    want = _weno64(method, x.astype(np.float64))
    for got, ref in zip((r, l), want):
        err = (got.cpu().numpy().astype(np.float64) - ref) * 2.0 ** 23
        assert np.max(np.abs(err)) <= 6.0
        assert np.sqrt(np.mean(err ** 2)) <= 0.3
