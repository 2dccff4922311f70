"""The F-K step of the gather resampling (rtm_fk.cuh) against numpy's double-precision FFT form of
the same steps, over lengths where its power-of-two convolutions, frequency counts and the change to
the library transforms can go wrong."""
import numpy as np
import pytest


def _fk(obs, nx, lx, mirror):
    """General F-K interpolation, GeneralFKinterp (Interp_function.cpp:53-244), in 64 bits."""
    nt0, nx0 = obs.shape
    a = obs.T.astype(np.float64)
    nf = 1 + nt0 // 2
    K = np.fft.fft2(a)[:, :nf]
    S = np.fft.fft2(a, s=(lx * nx0, lx * nt0))
    Z = S.reshape(lx, nx0, lx * nt0).sum(0) / lx
    H = S[:, :nf] / np.tile(Z[:, :nf] + np.float32(np.abs(Z).max()) * 1e-5, (lx, 1))
    H = np.where(np.abs(H) > lx * lx, lx, H)
    g = np.fft.ifft(H * np.tile(K, (lx, 1)), axis=0, norm="forward")[:nx]
    G = np.zeros((nx, nt0), complex)
    G[:, :nf] = g
    for k in range(nf, nt0):
        src = nt0 - k if mirror else (nt0 + 1) // 2 - (k - nf)
        if src < nf:
            G[:, k] = g[:, src].conj()
    return np.fft.ifft(G, axis=1, norm="forward").real.T


# lengths: the shortest, powers of two and their neighbours, primes, even and odd sample counts, the
# longest of the own transforms (4096 samples, 4096 padded traces) and one past each (library
# transforms); folds 2 to 5
@pytest.mark.gpu
@pytest.mark.parametrize("nx0,nt0,lx", [(2, 4, 2), (3, 5, 2), (8, 16, 3), (9, 17, 2), (16, 33, 4), (61, 617, 2),
                                        (241, 500, 2), (127, 1024, 3), (129, 1025, 5), (40, 4096, 2), (40, 4097, 2),
                                        (1024, 64, 4), (1025, 64, 4)])
@pytest.mark.parametrize("mirror", [0, 1])
def test_fk_step_matches_double_precision_fft(rtmlib, nx0, nt0, lx, mirror):
    rng = np.random.default_rng(nx0 * nt0)
    t, x = np.arange(nt0)[:, None], np.arange(nx0)[None, :]
    obs = 0.01 * rng.standard_normal((nt0, nx0))
    for k in range(4):
        u = 0.35 * (t - nt0 * (k + 1) / 5 - 0.2 * k * x)
        obs = obs + (1 - 2 * u * u) * np.exp(-u * u)
    obs = obs.astype(np.float32)
    nx = lx * (nx0 - 1) + 1
    got = rtmlib.interp_gather(obs, nx, nt0, 1e-3, 1e-3, mirror)   # nt == nt0: the F-K step alone
    want = _fk(obs, nx, lx, mirror)
    assert np.abs(want).max() > 0
    # float32 rounding of the result (6e-8) and of max|Z|; the double transforms' errors are 1e-12
    # of the largest value after the division by the near-zero folds
    assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
