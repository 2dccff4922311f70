"""Kept workspaces of the gather resampling (rtm_interp.cu) beside other shapes and callers."""
import threading

import numpy as np
import pytest


def _survey(G, nx, nt):
    return G.SurveyConfig(nx=nx, nz=60, nt=nt, dx=10.0, dz=10.0, dt=float(np.float32(1e-3)), npml=12, fdom=25.0,
                          layout=2, spx0=100.0, spz0=20.0, dspx=10.0, mode=1, mute=0)


def _models(nx):
    return np.full((60, nx), 2000, np.float32), np.full((60, nx), 2000, np.float32)


def _record(nt0, nx0, seed):
    return np.random.default_rng(seed).standard_normal((nt0, nx0)).astype(np.float32)


# a session's kept plan of the longest transforms, then a shorter shape's plan (alone, and another
# session's), then the kept one again: transforms of 8192, 4096 and 1024 points against 128
@pytest.mark.gpu
@pytest.mark.parametrize("nt0", [4096, 1500, 500])
def test_a_kept_plan_survives_a_shorter_one(rtmlib, nt0):
    G = rtmlib
    nx0, nx = 61, 121
    v, rho = _models(nx)
    obs, short = _record(nt0, nx0, nt0), _record(60, 10, 1)
    with G.Session(_survey(G, nx, nt0), G.RunOptions(), [1], v, rho) as ss:
        ss.set_gather_raw(0, obs, 1e-3)
        want = ss.gather(0)
        assert np.abs(want).max() > 0
        G.interp_gather(short, 19, 60, 1e-3, 1e-3)
        ss.set_gather_raw(0, obs, 1e-3)
        assert np.array_equal(ss.gather(0), want)
        vs, rs = _models(19)
        with G.Session(_survey(G, 19, 60), G.RunOptions(), [1], vs, rs) as other:
            other.set_gather_raw(0, short, 1e-3)
            ss.set_gather_raw(0, obs, 1e-3)
        assert np.array_equal(ss.gather(0), want)


@pytest.mark.gpu
def test_plans_of_two_lengths_in_two_threads(rtmlib):
    G = rtmlib
    shapes = [(1500, 41, 81), (60, 10, 19)]
    want = [G.interp_gather(_record(nt0, nx0, nt0), nx, nt0, 1e-3, 1e-3) for nt0, nx0, nx in shapes]
    errors = []

    def work(k):
        nt0, nx0, nx = shapes[k]
        obs = _record(nt0, nx0, nt0)
        try:
            for _ in range(40):
                assert np.array_equal(G.interp_gather(obs, nx, nt0, 1e-3, 1e-3), want[k])
        except Exception as e:   # (a thread's failure must reach the test)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
