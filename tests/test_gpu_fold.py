"""The fold of a row longer than its channel: one rounded twiddle per value.

With a single nonzero at (0, c) a row of S is the chirp at c alone, and channel
q's buffer holds that value times one twiddle W_L^{qc} in slot c mod Lp.  The
mean of output / exact output over the row is 1 + (1/K) * the sum of the
channels' relative errors at that one value, plus what the network adds to the
slot: rounded twiddles, the same for every column of that slot.  The column
c mod Lp, which does not fold, has that part alone (and its own rounded
entries), so the difference of the two means holds the fold's; what else
differs from output to output averages out (1e-9), but for the roundings of the
first stage's products (about 24 at 3e-8, so 6e-9, independent from column to
column).

The columns are those where a product of two rounded twiddles
W_L^{qn} * W_K^{qj} would shift the mean most (2e-8 and more).  Regressing the
measured means, less what the single rounded entries explain, on that shift
gives 0 for one entry per value and 1 for the product of two; with 24 columns
6e-9 of noise moves the coefficient by 6e-9 / 2e-8 / sqrt(24) = 0.06, so the
bar of 0.4 is six such steps from both.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb

pytestmark = pytest.mark.gpu


def f32(z):
    return np.asarray(z.real, np.float32) + 1j * np.asarray(z.imag, np.float32).astype(np.float64)


def cmul(a, b):
    """FP32 complex product as the kernels form it (one rounded product, one FMA per part)."""
    def r(x):
        return np.asarray(x, np.float32).astype(np.float64)
    re = r(a.real * b.real + r(-a.imag * b.imag))
    im = r(a.real * b.imag + r(a.imag * b.real))
    return re + 1j * im


def root(e, n):
    return np.exp(-2j * np.pi * (e % n) / n)


@pytest.mark.parametrize("cols,kw", [(40421, dict(length_policy=7)), (40421, dict(length_policy=2)),
                                     (11003, dict(length_policy=7, max_channel_len=2800)),
                                     (40421, dict(length_policy=7, channel_mode=1))])
def test_fold_rounds_one_twiddle(cuda, cols, kw):
    import torch

    def plan(c):
        coo = gb.COOMatrix(5, cols, np.zeros(1, np.int32), np.full(1, c, np.int32))
        return gb.Plan(coo, **kw)

    with plan(0) as p:
        L, K, Lp = p.info["fft_len"], p.info["channels"], p.info["channel_len"]
    assert K > 2 and cols > Lp
    c = np.random.default_rng(cols).permutation(np.arange(Lp, cols))[:4000].astype(np.int64)
    assert np.all(c // Lp >= 1)

    def errors(c):
        """Relative error of the mean with one entry per value, and with a product of two."""
        chirp = np.exp(-1j * np.pi * (c * c % (2 * cols)) / cols)
        x = f32(chirp)
        one, two = np.zeros(c.size, np.complex128), np.zeros(c.size, np.complex128)
        for q in range(K):
            exact = chirp * root(q * c, L)
            a = cmul(x, f32(root(q * c, L))) if q else x
            b = cmul(cmul(x, f32(root(q * (c // Lp * Lp), L))), f32(root(q * (c % Lp), L))) if q else x
            one += (a / exact - 1) / K
            two += (b / exact - 1) / K
        return one, two

    v = np.arange(cols // 2 + 1, dtype=np.int64)

    def mean(c):
        with plan(int(c)) as p:
            out = p.empty_output()
            p.execute(out)
            torch.cuda.synchronize()
            assert p.error_flags() == 0
            got = out[0, :v.size].cpu().numpy().astype(np.complex128)
        return np.mean(got * np.conj(root(v * c, cols))) - 1

    one, two = errors(c)
    slot = errors(c % Lp)[0]
    shift = two - one
    pick = np.argsort(-np.abs(shift))[:24]
    assert np.abs(shift[pick]).min() > 2e-8
    coef = sum(np.real(np.conj(shift[i]) * (mean(c[i]) - one[i] - (mean(c[i] % Lp) - slot[i]))) for i in pick)
    coef /= np.sum(np.abs(shift[pick]) ** 2)
    assert abs(coef) < 0.4, f"{coef:.2f} (1: a product of two rounded twiddles)"
