"""Host check of the g(r) bin estimate (gr_bins, gr_estimate and the settle band
in csrc/gr_bins.cuh, gr_with_shift in csrc/gder.cu), restated in numpy float32.

A pair whose estimate is not left open must fall in the reference's bin
(get_gder.cu:113-121), and a pair whose estimated squared distance reaches
`near` must be out of range, for distances spread over the range and packed
around every bin edge, with the approximate reciprocal square root off by up to
2^-22.9 either way, and for pairs across the faces of the box, where the
kernel's shifted position and the reference's difference round differently."""
import os
import re

import numpy as np
import pytest

F, D = np.float32, np.float64
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bd_aging_b200", "csrc")


def constant(name, pattern):
    with open(os.path.join(CSRC, name)) as f:
        return float(re.search(pattern, f.read()).group(1))


C1 = constant("gr_bins.cuh", r"kGrC1 = ([0-9.e-]+)f")
SHIFT = constant("gder.cu", r"err = ([0-9.e-]+)f \* side")


def fma(a, b, c):  # products of two floats are exact in double
    return (a.astype(D) * D(b) + D(c) if np.ndim(b) == 0 else a.astype(D) * b.astype(D) + np.asarray(c, D)).astype(F)


def ref_bin(d2, rng, nbins):
    """Bin of a rounded squared distance by the reference's rule, -1 out of range."""
    bs = F(rng) / F(nbins)
    dist = np.sqrt(d2)
    b = (dist / bs).astype(np.int64)
    return np.where(dist < F(rng), np.where(b == nbins, nbins - 1, b), -1)


class Bins:
    """gr_bins, then gr_with_shift for a box of side L."""

    def __init__(self, rng, nbins, L=None):
        lo, hi = 0, 0x7F800000
        while lo < hi:
            mid = lo + (hi - lo) // 2
            if not np.sqrt(np.array([mid], np.uint32).view(F)[0]) < F(rng):
                hi = mid
            else:
                lo = mid + 1
        self.thr = np.array([lo], np.uint32).view(F)[0]
        self.inv_bin = F(1) / (F(rng) / F(nbins))
        self.near = F(D(self.thr) * (1 + 1.2e-6))
        self.c0 = F(1e-6)
        if L is not None:
            err = F(SHIFT) * F(L)
            f = F(1) + err / F(rng)
            self.near = self.near * (f * f)
            self.c0 = self.c0 + F(1.1) * err * self.inv_bin

    def estimate(self, d2, rel):
        """Bin and whether it stays open; the reciprocal square root off by `rel`."""
        r = (1 / np.sqrt(d2.astype(D)) * (1 + rel)).astype(F)
        q = fma((d2 * r).astype(F), self.inv_bin, -0.5)
        qm = np.rint(q)  # adding and taking back 1.5 2^23
        h = fma(q, F(-C1), F(F(0.5) - F(C1) - self.c0))
        return qm.astype(np.int64), ~(np.abs(q - qm) <= h)


def check(d2_est, d2_ref, rng, nbins, bins):
    want = ref_bin(d2_ref, rng, nbins)
    out = d2_est >= bins.near
    assert np.all(want[out] == -1)
    for rel in (0.0, 2.0 ** -22.9, -(2.0 ** -22.9)):
        b, open_ = bins.estimate(d2_est, rel)
        closed = ~out & ~open_
        got = np.where(b < nbins, b, -1)  # a slot past the last bin is not counted
        np.testing.assert_array_equal(got[closed], want[closed])
    return np.mean(~out & bins.estimate(d2_est, 0.0)[1])


def sums(d):  # fused as the kernels add them, and rounded as the reference does
    fused = fma(d[2], d[2], fma(d[1], d[1], (d[0] * d[0]).astype(F)))
    return fused, ((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]).astype(F)


def distances(g, rng, nbins, n):
    """Uniform over the range, and at every bin edge within 4e-6 of it."""
    edge = rng / nbins * np.arange(1, nbins + 1)
    near = (edge[:, None] * (1 + 4e-6 * g.uniform(-1, 1, (nbins, max(1, n // nbins))))).ravel()
    return np.concatenate([g.uniform(0.01, 1.02, n) * rng, near])


@pytest.mark.parametrize("rng,nbins", [(15.0, 400), (3.0, 300), (2.5, 64), (5.0, 200), (0.7, 1), (6.1, 4096)])
def test_closed_estimates_are_the_reference_bins(rng, nbins):
    g = np.random.default_rng(nbins)
    r = distances(g, rng, nbins, 200000)
    u = g.normal(size=(3, len(r)))
    d = [(c * r / np.sqrt((u ** 2).sum(0))).astype(F) for c in u]
    est, ref = sums(d)
    assert check(est, ref, rng, nbins, Bins(rng, nbins)) < 0.6


@pytest.mark.parametrize("L,rng,nbins", [(29.3, 12.0, 400), (53.0, 21.0, 300), (8.1, 2.0, 64), (101.6, 15.0, 4096)])
def test_closed_estimates_across_faces_are_the_reference_bins(L, rng, nbins):
    """x_i in the box, x_j across one to three of its faces."""
    g = np.random.default_rng(nbins)
    L = F(L)
    r = distances(g, rng, nbins, 100000)
    u = np.abs(g.normal(size=(3, len(r)))) + 0.05
    d = u * r / np.sqrt((u ** 2).sum(0))
    across = g.random((3, len(r))) < 0.7
    est, ref = [], []
    for c in range(3):
        # the image at x_i + d lies in (L, 1.5 L) where the pair crosses this face
        xi = np.where(across[c], L - g.random(len(r)) * np.minimum(d[c], L / 2), g.random(len(r)) * (L - d[c])).astype(F)
        xj = np.where(across[c], xi.astype(D) + d[c] - D(L), xi.astype(D) + d[c]).astype(F)
        s = np.where(across[c], L, F(0))
        est.append((xi - (xj + s)).astype(F))
        ref.append(((xi - xj).astype(F) - s).astype(F))
    (e2, _), (_, r2) = sums(est), sums(ref)
    check(e2, r2, rng, nbins, Bins(rng, nbins, L))


@pytest.mark.parametrize("L,lo,hi", [(53.48, 10.6, 26.0), (45.17, 18.9, 22.0), (33.0, 0.5, 15.0),
                                     (16.25, 0.2, 8.0), (31.99, 0.02, 15.0)])
def test_shift_bound_covers_both_roundings(L, lo, hi):
    """The kernel rounds x_j + s and the reference x_i - x_j, half an ulp each, in
    up to three components.  Coordinates fall on the grid of half an ulp of the
    sums now and then, where ties round the two apart."""
    assert SHIFT >= np.sqrt(3.0) * 2.0 ** -24 * 2.0
    g = np.random.default_rng(int(L))
    L = F(L)
    d = g.uniform(lo, hi, 1000000)
    x = (g.random(len(d)) ** 2 * lo * 0.98).astype(F)
    for xi, s in (((L - x).astype(F), L), (x, -L)):
        xj = (xi.astype(D) + np.sign(s) * d - D(s)).astype(F)
        image = xj + s
        ok = (xj >= 0) & (xj <= L) & (xi <= L) & (image <= F(1.5) * L) & (image >= F(-0.5) * L)
        gap = np.abs((xi - image).astype(D) - ((xi - xj) - s).astype(D))[ok]
        ulps = (np.spacing(np.abs(image)) + np.spacing(np.abs(xi - xj)) + np.spacing(np.abs(xi - image)))[ok]
        assert len(gap) > 1000 and np.all(gap <= ulps.astype(D) / 2)
        assert np.sqrt(3.0) * gap.max() <= SHIFT * L
