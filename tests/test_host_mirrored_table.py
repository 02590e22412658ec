"""d^l_{m,-n}(beta) = (-1)^(l + m) d^l_{m,n}(pi - beta) in the reference recursion: where it holds, and where it is relied on.

The rule of the tensor-core plans (small batches share table rows between the groups (m0, +-n0)): the smallest seed on the grid,
cos(beta / 2)^(2 l) at beta = pi - pi / (2 N), is a normal double.  Bound: 1e-12, a thousandth of the FP32-data plans' error of a
sum of 2 l terms.
"""
import math

import numpy as np
import pytest


def relied_on(L):
    return 2.0 * L * math.log2(math.sin(math.pi / (4.0 * (2 * L + 2)))) > -1022.0


def difference(oracle, L, ks):
    worst = 0.0
    for k in ks:
        a, b = (oracle.wigner_d(oracle.beta_k(L, j), L) for j in (k, 2 * L + 1 - k))
        for l in range(L + 1):
            o, W = l * (4 * l * l - 1) // 3, 2 * l + 1
            A, B = (x[o:o + W * W].reshape(W, W).T for x in (a, b))  # [m, n]
            sg = (-1.0) ** (l + np.arange(-l, l + 1))
            worst = max(worst, float(np.abs(A[:, ::-1] - sg[:, None] * B).max()))
    return worst


@pytest.mark.parametrize("L", [1, 2, 7, 31, 60, 66, 67, 68])
def test_mirrored_where_relied_on(oracle, L):
    assert relied_on(L)
    assert difference(oracle, L, range(2 * L + 2)) <= 1e-12


@pytest.mark.parametrize("L", [72, 96, 127])
def test_not_mirrored_where_not(oracle, L):
    assert not relied_on(L)
    assert difference(oracle, L, [0, 1]) > 0.5


def test_limit():
    assert [L for L in range(512) if relied_on(L)] == list(range(69))
