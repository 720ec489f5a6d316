"""The sequences that replace CUDA's FP64 square roots and divisions in the solver and the grid lookups, against the
operations themselves, bit for bit: random operands over all exponents, the edges of the ranges in which a sequence is
used, zeros, subnormals, infinities and NaN, mantissas of all ones, and the operands whose exact result lies closest to
halfway between two doubles (found by modular arithmetic), where a sequence that is not exact would round wrongly."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def device_fn(tmp_path_factory):
    import torch
    from rainbow_b200 import build as B
    out = str(tmp_path_factory.mktemp("rounding") / "rounding.so")
    subprocess.check_call([os.environ.get("NVCC", "nvcc")] + B.NVCC_FLAGS +
                          ["-I", os.path.join(B.HERE, "csrc"), "-o", out, os.path.join(HERE, "rounding.cu")])
    fn = ctypes.CDLL(out).rounding
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_int]

    def call(what, a, b):
        ta, tb = (torch.from_numpy(np.ascontiguousarray(v, np.float64)).cuda() for v in (a, b))
        to = torch.empty_like(ta)
        assert fn(what, ta.data_ptr(), tb.data_ptr(), to.data_ptr(), len(a)) == 0
        return to.cpu().numpy()
    return call


def _same(got, want, *operands):
    with np.errstate(all="ignore"):
        bad = ~((got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want)))
    assert not bad.any(), [(v[bad][:4], ) for v in operands + (got, want)] + [int(bad.sum())]


def _special():
    """Pairs of values at the edges of everything."""
    tiny, eps = np.finfo(float).tiny, 2.0 ** -52
    v = [0.0, np.inf, np.nan, tiny, tiny * eps, 3 * tiny * eps, np.finfo(float).max]
    for e in (-1022, -1021, -501, -500, -499, -401, -400, -399, -1, 0, 1, 2, 399, 400, 401, 499, 500, 501, 1022, 1023):
        v += [2.0 ** e * m for m in (1.0, 1.0 + eps, 1.5, 2.0 - eps, 2.0 - 2 * eps)]
    v = np.array(v + [-x for x in v])
    return [w.ravel() for w in np.meshgrid(v, v)]


def _random(rng, n, lo, hi):
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n) * rng.choice([-1.0, 1.0], n)


def _hard_divisions(divisors, far=5):
    """For divisors of mantissa D / 2^52 (D odd), the dividends n whose quotient lies k / (2^53 D), |k| <= far, from a
    point halfway between two doubles: 2^53 A - M D = k with n = A / 2^52 and the halfway point M / 2^53."""
    out = []
    for D in divisors:
        inverse = pow(int(D), -1, 1 << 53)
        for k in [k for k in range(-far, far + 1) if k]:
            M = (-k * inverse) % (1 << 53) + (1 << 53)
            A = (M * int(D) + k) >> 53
            if A < 1 << 53 or (A < 1 << 54 and A % 2 == 0):
                out.append((A * 2.0 ** -52, int(D) * 2.0 ** -52))
    return np.array(out).T


def _odd_mantissas(rng, n):
    """Random ones, and those next to a power of two from both sides."""
    near = np.arange(1, 400, 2)
    return np.concatenate([rng.integers(1 << 51, 1 << 52, n) * 2 + 1, (1 << 53) - near, (1 << 52) + near])


def _hard_squares(far=4096):
    """The values of [1, 4) whose root lies closest to halfway between two doubles: odd M in (2^53, 2^54) with M^2 within
    `far` of a multiple of 2^54 (of 2^55 for values from 2 up), by lifting the roots of c modulo powers of two."""
    out = []
    for c in range(-far, far + 1):
        if c % 8 != 1:   # an odd square
            continue
        roots = [1, 3, 5, 7]          # modulo 8, then modulo 16, 32, ...
        for bits in range(4, 56):
            roots = [x for r in roots for x in (r, r + (1 << (bits - 1))) if (x * x - c) % (1 << bits) == 0]
            for M in roots if bits in (54, 55) else []:
                A = (M * M - c) >> bits
                if (1 << 53) < M < (1 << 54) and (1 << 52) <= A < (1 << 53):
                    out.append(A * 2.0 ** (bits - 106))
    return np.unique(out)


def test_ratio_sqrt(device_fn):
    rng = np.random.default_rng(0)
    squares = _hard_squares()
    assert len(squares) > 1000 and squares.min() >= 1.0 and squares.max() < 4.0
    ones = 4.0 - 2.0 ** -51 * np.arange(0, 400)      # roots whose mantissas are all ones, or nearly
    roots = np.concatenate([squares, ones, rng.uniform(1.0, 1.0 + 2.0 ** -30, 4000) ** 2, rng.uniform(1.0, 4.0, 4000)])
    # dividends of 1, of the root itself, and the worst ones for each root as a divisor
    a, v = [np.ones(len(roots)), np.sqrt(roots), 2.0 - 2.0 ** -52 + 0 * roots], [roots] * 3
    D = (np.sqrt(roots) * 2.0 ** 52).astype(np.int64)
    for r, d in zip(roots, D):
        if d % 2 and d < 1 << 53:
            n, _ = _hard_divisions([d])
            a.append(n)
            v.append(np.full(len(n), r))
    a, v = np.concatenate(a), np.concatenate(v)
    scale = rng.integers(-240, 240, (2, len(a)))
    a, v = np.concatenate([a, a * 2.0 ** scale[0]]), np.concatenate([v, v * 4.0 ** scale[1]])
    s = _special()
    n = 1 << 20
    a = np.concatenate([a, s[0], _random(rng, n, -1022, 1023), _random(rng, n, -3, 3)])
    v = np.concatenate([v, s[1], np.abs(_random(rng, n, -1022, 1023)), np.abs(_random(rng, n, -3, 3))])
    with np.errstate(all="ignore"):
        _same(device_fn(0, a, v), a / np.sqrt(v), a, v)


def test_quotient(device_fn):
    rng = np.random.default_rng(1)
    n, d = _hard_divisions(_odd_mantissas(rng, 20000))
    scale = rng.integers(-300, 300, (2, len(n)))
    n, d = np.concatenate([n, n * 2.0 ** scale[0]]), np.concatenate([d, d * 2.0 ** scale[1]])
    s = _special()
    m = 1 << 20
    # dividends and remainders next to the subnormal range, divisors whose reciprocal is
    small = _random(rng, m, -1074, -950), _random(rng, m, -220, -160)
    large = _random(rng, m, 0, 1023), _random(rng, m, 1000, 1023)
    n = np.concatenate([n, s[0], _random(rng, m, -1022, 1023), _random(rng, m, -3, 3), small[0], large[0]])
    d = np.concatenate([d, s[1], _random(rng, m, -1022, 1023), _random(rng, m, -3, 3), small[1], large[1]])
    with np.errstate(all="ignore"):
        _same(device_fn(1, n, d), n / d, n, d)


def test_sqrt_chain(device_fn):
    """Right to half a unit in the last place and the ~2^-23 of one that its last correction leaves: the rounded root on all
    but a 2^-22 share of operands, and never further off than its neighbour."""
    rng = np.random.default_rng(2)
    squares = _hard_squares()
    v = np.concatenate([squares, 4.0 - 2.0 ** -51 * np.arange(0, 400), rng.uniform(1.0, 4.0, 1 << 20)])
    v = np.concatenate([v, v * 4.0 ** rng.integers(-500, 500, len(v))])
    got, want = device_fn(2, v, v), np.sqrt(v)
    assert np.abs(got.view(np.int64) - want.view(np.int64)).max() <= 1
    assert (got != want).sum() <= 2 * (len(squares) + 400) + 8
    assert np.isnan(device_fn(2, np.zeros(1), np.zeros(1))).all()
