"""Rounding of the Biot-Savart kernel's own square root and quotient, alone and inside the kernel."""

import ctypes
import random
import subprocess

import numpy as np
import pytest

from snoopy_b200 import _lib, fem_c

pytestmark = pytest.mark.gpu


def _roots(a, b):
    import torch

    a, b = (torch.as_tensor(np.ascontiguousarray(v)).cuda() for v in (a, b))
    out = torch.empty(2, a.numel(), dtype=torch.float64, device="cuda")
    _lib.call("snp_biot_savart_roots", a.numel(), _lib.ptr(a), _lib.ptr(b), _lib.ptr(out[0]), _lib.ptr(out[1]),
              _lib.stream_ptr())
    return out.cpu().numpy()


def _random(rng, n, lo, hi):
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


def _hard_quotients(n, seed):
    """n, d with n 2^k = M d + c, M a 54-bit odd integer, |c| small: n / d is c / d half-ulps from the
    middle of two doubles, as close as a quotient can be."""
    rng, out = random.Random(seed), []
    while len(out) < n:
        d, c, k = rng.randrange(2 ** 52, 2 ** 53) | 1, rng.choice([-1, 1, -3, 3, 5, -5, 7, -7]), rng.choice([53, 54])
        m = -c * pow(d, -1, 2 ** k) % 2 ** k + (2 ** 53 if k == 53 else 0)
        num = m * d + c
        if m % 2 and 2 ** 53 <= m < 2 ** 54 and num % 2 ** k == 0 and 0 < num >> k < 2 ** 53:
            out.append((float(num >> k), float(d)))
    return np.array(out).T


def _hard_roots(c_max):
    """Doubles a = M^2 - c, M a 54-bit odd integer, c = 1 mod 8 small: sqrt(a) is c / M half-ulps from the
    middle of two doubles."""
    out = set()
    for c in [*range(1, c_max, 8), *range(-7, -c_max, -8)]:
        roots = {1, 3, 5, 7}  # of c modulo 2^bits, lifted bit by bit
        for bits in range(3, 55):
            roots = {y % 2 ** bits for x in roots for y in (x, x + 2 ** (bits - 1)) if (y * y - c) % 2 ** (bits + 1) == 0}
        for s in roots:
            for m in (s % 2 ** 54, -s % 2 ** 54, s % 2 ** 53 + 2 ** 53, -s % 2 ** 53 + 2 ** 53):
                a = m * m - c
                if m % 2 and 2 ** 53 <= m < 2 ** 54 and a % 2 ** (a.bit_length() - 53) == 0:
                    out.add(float(a))
    return np.array(sorted(out))


@pytest.mark.parametrize("kind", ["random", "window", "squares", "hard", "ones"])
def test_root_and_quotient_round_as_ieee(kind):
    """Bit for bit numpy's (IEEE) results: random operands, the ends of the divisors' range, squares and
    their neighbours, operands whose results lie next to the middle of two doubles, and divisors with a
    significand of ones."""
    rng = np.random.default_rng(1)
    n = 1 << 20
    if kind == "random":
        a, b = _random(rng, n, -250, 250), _random(rng, n, -250, 250)
    elif kind == "window":
        a = _random(rng, n, -200, 200)
        b = _random(rng, n, -770, 770)
        b[:8] = np.ldexp([1.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), 1.5] * 2, [-767] * 4 + [769] * 4)
    elif kind == "squares":
        g = _random(rng, n, -400, 400)
        a = ((g * g).view(np.int64) + rng.integers(-2, 3, n)).view(np.float64)
        b = g
    elif kind == "hard":
        a, b = _hard_quotients(100000, 5)
        r = _hard_roots(20000)
        assert len(r) > 5000
        a, b = (np.concatenate(v) for v in ((a, r, r * 2.0 ** -400), (b, r, r)))
    else:
        j = rng.integers(0, 3, n)
        b = np.ldexp((np.full(n, np.nextafter(2.0, 0.0)).view(np.int64) - j).view(np.float64), rng.integers(-300, 300, n))
        a = np.where(rng.integers(0, 2, n) == 0, 1.0, rng.uniform(1.0, 2.0, n))
    root, quotient = _roots(a, b)
    assert np.array_equal(root, np.sqrt(a))
    assert np.array_equal(quotient, a / b)


_PLAIN = r"""
#include <math.h>
#include <stdint.h>
static double dot(const double *a, const double *b) { return fma(a[2], b[2], fma(a[0], b[0], a[1] * b[1])); }
static double minor2(double a, double b, double c, double d) { return fma(a, b, -(c * d)); }
void field(const double *src, int64_t n_src, const double *tar, int64_t n_tar, double current, double *B) {
    for (int64_t i = 0; i < n_tar; ++i) {
        double s[3] = {0.0, 0.0, 0.0};
        for (int64_t j = 0; j < n_src; ++j) {
            double a[3], b[3];
            for (int k = 0; k < 3; ++k) {
                a[k] = src[6 * j + k] - tar[3 * i + k];
                b[k] = src[6 * j + 3 + k] - tar[3 * i + k];
            }
            const double na = sqrt(dot(a, a)), nb = sqrt(dot(b, b)), pr = na * nb;
            const double f = (na + nb) / ((pr + dot(a, b)) * pr);
            s[0] += minor2(a[1], b[2], a[2], b[1]) * f;
            s[1] += minor2(a[2], b[0], a[0], b[2]) * f;
            s[2] += minor2(a[0], b[1], a[1], b[0]) * f;
        }
        for (int k = 0; k < 3; ++k) B[3 * i + k] = s[k] * current * 1e-7;
    }
}
"""


@pytest.mark.parametrize("n_src", [1, 128, 131])
def test_field_has_the_bits_of_the_plain_form(n_src, tmp_path):
    """Targets outside every filament's core, some of them just outside: the kernel against the same
    roundings with the C library's square root and the compiler's division."""
    (tmp_path / "plain.c").write_text(_PLAIN)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "plain.c", "-o", "plain.so", "-lm"],
                   cwd=tmp_path, check=True)
    plain = ctypes.CDLL(str(tmp_path / "plain.so")).field
    rng = np.random.default_rng(n_src)
    rad = 0.02
    a = rng.uniform(-1, 1, (n_src, 3))
    src = np.concatenate([a, a + rng.normal(0, 0.3, (n_src, 3))], axis=1)
    tar = rng.uniform(-1.5, 1.5, (20000, 3))
    k, axis = np.arange(2000), None
    j = rng.integers(0, n_src, len(k))
    axis = src[j, 3:] - src[j, :3]
    off = np.cross(axis, rng.normal(size=(len(k), 3)))
    off *= (rad * rng.choice([1.00005, 1.0002, 1.001, 1.5], len(k)) / np.linalg.norm(off, axis=1))[:, None]
    tar[k] = src[j, :3] + rng.uniform(-0.5, 1.5, len(k))[:, None] * axis + off
    # the distance of every target from every segment, for the targets inside a core
    inside = np.zeros(len(tar), bool)
    for s in src:
        n = s[3:] - s[:3]
        t = np.clip(((tar - s[:3]) @ n) / (n @ n), 0.0, 1.0)
        inside |= np.linalg.norm(tar - s[:3] - t[:, None] * n, axis=1) < rad * 1.00001
    tar = np.ascontiguousarray(tar[~inside])
    want = np.empty_like(tar)
    d = ctypes.c_double
    p = ctypes.POINTER(d)
    plain.argtypes = [p, ctypes.c_int64, p, ctypes.c_int64, d, p]
    plain.restype = None
    plain(src.ctypes.data_as(p), n_src, tar.ctypes.data_as(p), len(tar), 250.0, want.ctypes.data_as(p))
    got = fem_c.compute_B_line_segs_cpp(src, tar, 250.0, rad)
    assert len(tar) > 10000 and np.array_equal(got, want)
