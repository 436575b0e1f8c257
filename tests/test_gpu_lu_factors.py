"""The coarse LU, its explicit inverse and the banded substitution on matrices that pivot.

The multigrid's coarse matrices are diagonally heavy: they interchange few rows, those of
bands up to kl = 34 none.  Here the bands are random: normal values (nearly every step
interchanges, at every distance) and small integers (ties for the largest entry, zero
multipliers), the latter also with columns of zeros (zero pivots), at both sides of every
kernel's limits (kl = 20 one CTA; 32, 96, 224 and 480 the panels' block sizes; 240 and 496
the substitution's), with last panels of one column, in between and full.  Factors, pivots,
the first zero pivot, the inverse and the solutions equal, bit for bit, those of dgbtf2 and
dgbtrs (LAPACK's unblocked loops, written out below: one multiply and one add at a time).
"""
import numpy as np
import pytest

from tests import kernel_entries

pytestmark = pytest.mark.gpu


def dgbtf2(AB, n, kl, ku):
    kv = kl + ku
    ipiv = np.zeros(n, np.int32)
    info, ju = 0, 0
    for j in range(n):
        km = min(kl, n - 1 - j)
        jp = int(np.argmax(np.abs(AB[kv:kv + km + 1, j])))
        ipiv[j] = jp + j + 1
        if AB[kv + jp, j] == 0.0:
            info = info or j + 1
            continue
        ju = max(ju, min(j + ku + jp, n - 1))
        c = np.arange(j, ju + 1)
        r = kv - (c - j)  # row j of these columns
        if jp:
            AB[r, c], AB[r + jp, c] = AB[r + jp, c], AB[r, c]
        if km:
            l = AB[kv + 1:kv + km + 1, j] * (1.0 / AB[kv, j])
            AB[kv + 1:kv + km + 1, j] = l
            top = AB[r[1:], c[1:]]
            on = top != 0.0
            rr = r[1:][on][None, :] + np.arange(1, km + 1)[:, None]
            AB[rr, c[1:][on][None, :]] += l[:, None] * -top[on][None, :]
    return ipiv, info


def dgbtrs(AB, ipiv, n, kl, ku, B):
    """In place on the columns of B."""
    kv = kl + ku
    for j in range(n - 1):
        lm = min(kl, n - 1 - j)
        p = ipiv[j] - 1
        if p != j:
            B[[j, p]] = B[[p, j]]
        t = -B[j]
        on = t != 0.0
        B[j + 1:j + 1 + lm, on] += AB[kv + 1:kv + 1 + lm, j][:, None] * t[on][None, :]
    for j in range(n - 1, -1, -1):
        on = B[j] != 0.0
        t = B[j, on] / AB[kv, j]
        B[j, on] = t
        i0 = max(0, j - kv)
        B[i0:j, on] -= t[None, :] * AB[kv - j + i0:kv, j][:, None]


def band(kind, n, kl, ku, seed):
    rng = np.random.default_rng(seed)
    AB = np.zeros((2 * kl + ku + 1, n), order="F")
    v = rng.standard_normal((kl + ku + 1, n)) if kind == "normal" else rng.integers(-2, 3, (kl + ku + 1, n)) * 1.0
    for r in range(kl + ku + 1):  # band row kl + r holds row c + r - ku of column c
        c = np.arange(n)
        ok = (c + r - ku >= 0) & (c + r - ku < n)
        AB[kl + r, ok] = v[r, ok]
    if kind == "singular":
        AB[:, [n // 3, n // 3 + 1, n - 2]] = 0.0
    return AB


SIZES = [(160, 10), (297, 20), (97, 18), (200, 21), (273, 32), (160, 33), (299, 64), (311, 96), (320, 97), (449, 180),
         (480, 224), (500, 225), (700, 480), (70, 60), (620, 500)]


def in_matrix(n, kl, ku):
    r, c = np.meshgrid(np.arange(2 * kl + ku + 1), np.arange(n), indexing="ij")
    i = c + r - kl - ku
    return (i >= 0) & (i < n)


@pytest.mark.parametrize("kind", ["normal", "integer", "singular"])
@pytest.mark.parametrize("n,kl", SIZES)
def test_factors_and_inverse(gpu_lib, kind, n, kl):
    L = kernel_entries.load()
    ku = kl
    A = band(kind, n, kl, ku, n + kl)
    ref = A.copy(order="F")
    piv, info = dgbtf2(ref, n, kl, ku)
    assert np.count_nonzero(piv != np.arange(1, n + 1)) > n // 4
    assert info == (n // 3 + 1 if kind == "singular" else 0)
    m = in_matrix(n, kl, ku)
    for no_cluster in (0, 1):
        out = A.copy(order="F")
        p, inf = np.zeros(n, np.int32), np.zeros(2, np.int32)
        assert L.entry_lu(kernel_entries.ptr(out), n, kl, ku, kernel_entries.ptr(p), kernel_entries.ptr(inf), no_cluster) == 0
        assert (inf[0], inf[1]) == (info, 0)
        assert np.array_equal(p, piv)
        assert np.array_equal(out[m], ref[m])
    if info == 0:
        inv = np.zeros((n, n))
        assert L.entry_inverse(kernel_entries.ptr(ref), kernel_entries.ptr(piv), n, kl, ku, kernel_entries.ptr(inv)) == 0
        B = np.eye(n)
        dgbtrs(ref, piv, n, kl, ku, B)
        assert np.array_equal(inv, B)


@pytest.mark.parametrize("a,b,kl,fp32", [(20, 16, 20, 0), (30, 10, 97, 1), (40, 12, 200, 0), (30, 20, 240, 0),
                                         (30, 20, 241, 0), (36, 20, 496, 1), (36, 20, 497, 0), (8, 6, 30, 0)])
def test_substitution(gpu_lib, a, b, kl, fp32):
    L = kernel_entries.load()
    n, ku = (a + 1) * (b + 1), kl
    A = band("normal", n, kl, ku, n + kl)
    piv, info = dgbtf2(A, n, kl, ku)
    assert info == 0
    rng = np.random.default_rng(kl)
    rowb, rhs = rng.uniform(0.5, 2.0, n), rng.standard_normal(n)
    i, k = np.arange(n) // (b + 1), np.arange(n) % (b + 1)
    inner = (i > 0) & (i < a) & (k > 0) & (k < b)
    if fp32:
        rhs = rhs.astype(np.float32).astype(np.float64)
    B = np.where(inner, rhs * rowb, 0.0)[:, None]
    dgbtrs(A, piv, n, kl, ku, B)
    want = B[:, 0].astype(np.float32) if fp32 else B[:, 0]
    for no_cluster in (0, 1):
        x, to = np.zeros(n), np.zeros(1, np.int32)
        P = kernel_entries.ptr
        assert L.entry_solve(P(A), P(piv), P(rowb), a, b, kl, ku, P(rhs), P(x), fp32, no_cluster, P(to)) == 0
        assert to[0] == 0
        assert np.array_equal(x[inner], want[inner])
