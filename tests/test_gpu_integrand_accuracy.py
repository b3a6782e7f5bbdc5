"""W(lambda) by the sliced precisions against FP64: the digits of Y alone may limit it.

With W = sum_ij S_ij (Y Y^T)_ij, S the symmetric weights without their diagonal, rounding row i of Y to
multiples of u_i = 2^(e_i - 7 S) (e_i: exponent of its largest entry) moves W by
2 sum_iv d_iv (S Y)_iv with d_iv uniform in +-u_i/2: a standard deviation of
2 sqrt(sum_iv u_i^2/12 (S Y)_iv^2). The products that are dropped have to stay below that: over 60 samples
the root mean square of error/deviation is 1 with a spread of 0.09, and 1.5 is allowed. (In a numpy
emulation: 0.9 to 1.2; without the products t + u = S 3.7 for four slices and 5.0 for five, and
2 Y . (S Y), with the weights sliced too, 1.4 and 2.6.)"""
import numpy as np
import pytest
import torch

from gammcor_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [4, 5])
def test_integrand_error_is_that_of_the_digits(gpu_lib, S):
    n, nin, nact = 24, 4, 4
    nocc = nin + nact
    occ = np.r_[np.ones(nin), 0.95, 0.9, 0.1, 0.05, np.zeros(n - nocc)]
    indn = api.pair_space(occ, nin + 2)
    N, (p, q) = len(indn), (indn - 1).T
    c = np.where(occ >= 0.5, 1.0, -1.0) * np.sqrt(occ)
    g = np.digitize(np.arange(n), [nin, nocc])
    same = (g[p] == g[q])[:, None] & (g[p] == g[q]) & (g[p][:, None] == g[p])
    cc, rec = c[p] + c[q], p + q * n
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    eig = dev(np.ones(N))
    ratio = []
    for seed in range(60):
        rng = np.random.default_rng(seed)
        y = np.diag(rng.uniform(0.3, 0.8, N)) + 0.05 * rng.standard_normal((N, N))
        fofo = 0.05 * rng.standard_normal((n * nocc, n * nocc))
        k = np.where(same, 0.0, cc[:, None] * cc * fofo[np.ix_(rec, rec)])
        s = k + k.T
        np.fill_diagonal(s, 0.0)
        u = 2.0 ** (np.frexp(np.abs(y).max(1))[1] - 7 * S)
        sigma = 2 * np.sqrt(np.sum(u[:, None] ** 2 / 12 * (s @ y) ** 2))
        w = [api.ace_ne_erpa_fofo(dev(y.T).t(), eig, occ, indn, nact, nin, dev(fofo), precision=prec)
             for prec in ("fp64", f"fp64tc{S}")]
        ratio.append((w[1] - w[0]) / sigma)
    assert np.sqrt(np.mean(np.square(ratio))) < 1.5
