"""The pipelined stencil kernels (rtm_pipe.cu) against the one-column kernels (rtm_stencil.cu) at
the sizes where a tile, a stage or a list can go wrong, and the copies of results to the host.

Both forms round every operation alike, so all comparisons are exact."""
import ctypes as C

import numpy as np
import pytest


def _models(nz, nx, seed):
    rng = np.random.default_rng(seed)
    v = 1800 + 6 * np.arange(nz)[:, None] + 150 * rng.random((nz, nx))
    return np.minimum(v, 3800).astype(np.float32), (2000 + 100 * rng.random((nz, nx))).astype(np.float32)


def _survey(G, nx, nz, npml, nt, mode=0, **kw):
    d = dict(nx=nx, nz=nz, nt=nt, dx=10.0, dz=10.0, dt=float(np.float32(1e-3)), npml=npml, fdom=25.0, layout=2,
             spx0=(nx // 3) * 10.0, spz0=20.0, dspx=10.0, mode=mode, mute=0)
    d.update(kw)
    return G.SurveyConfig(**d)


def _both(monkeypatch, G, heights, run):
    out = []
    for k, h in zip(("VEL", "VEL_RECON", "PRES", "PRES_RECON"), heights):
        monkeypatch.setenv("RTM_B200_BZ_" + k, str(h))
    for form in ("scalar", "vector"):
        monkeypatch.setenv("RTM_B200_KERNELS", form)
        out.append(run())
    return out


def _same(a, b):
    for k in ("image1", "image2s", "illum"):
        assert np.abs(a[k]).max() > 0 and np.array_equal(a[k], b[k]), k
    for x, y in zip(a["gathers"], b["gathers"]):
        assert np.array_equal(x, y)


# padded widths one below, at and one above whole tiles of 128 columns, and partial last tiles of 1,
# 4 and 127 columns; depths that leave 1, 7, 8 and 15 rows in the last tile; interior tiles
# present (X >= 384); one height for all (merged launches) and mixed heights (separate ones)
@pytest.mark.gpu
@pytest.mark.parametrize("X,Z,npml,heights", [
    (384, 129, 20, (8, 8, 8, 8)), (383, 136, 20, (16, 16, 16, 16)), (385, 143, 21, (8, 8, 8, 8)),
    (388, 128, 23, (16, 8, 8, 16)), (511, 97, 10, (32, 32, 32, 32)), (513, 151, 32, (16, 16, 16, 16)),
    (400, 200, 37, (64, 64, 64, 64)), (129, 60, 12, (8, 8, 8, 8)), (60, 300, 15, (16, 16, 16, 16))])
def test_pipelined_form_at_tile_edges(rtmlib, monkeypatch, X, Z, npml, heights):
    G = rtmlib
    nx, nz = X - 2 * npml, Z - 2 * npml
    v, rho = _models(nz, nx, X + Z)
    s = _survey(G, nx, nz, npml, 90)
    _same(*_both(monkeypatch, G, heights, lambda: G.migrate(s, G.RunOptions(), [1, 3], v, rho)))


# every accumulator and strip type in both launch plans
@pytest.mark.gpu
@pytest.mark.parametrize("accum", [0, 1, 2, 3])
@pytest.mark.parametrize("heights", [(8, 8, 8, 8), (16, 16, 8, 8), (16, 16, 16, 16)])
def test_pipelined_form_of_every_type(rtmlib, monkeypatch, accum, heights):
    G = rtmlib
    nx, nz, npml = 391, 90, 18
    v, rho = _models(nz, nx, accum)
    s = _survey(G, nx, nz, npml, 70, receiver_depth=3)
    o = G.RunOptions(accum_fp64=accum, strip_precision=("fp32", "fp16", "bf16", "fp16")[accum],
                     gather_precision=("fp32", "bf16", "fp16", "fp32")[accum])
    _same(*_both(monkeypatch, G, heights, lambda: G.migrate(s, o, [1, 2], v, rho)))


# list lengths: fewer tiles than resident blocks, several per block (claimed from the counter), and
# more than 16 per block (every gridDim-th tile, every other launch backwards)
@pytest.mark.gpu
@pytest.mark.parametrize("shots", [1, 6, 24])
@pytest.mark.parametrize("heights", [(8, 8, 8, 8), (16, 16, 8, 8)])
def test_pipelined_form_for_short_and_long_tile_lists(rtmlib, monkeypatch, shots, heights):
    G = rtmlib
    nx, nz, npml = 350, 960, 20
    v, rho = _models(nz, nx, shots)
    s = _survey(G, nx, nz, npml, 40)
    _same(*_both(monkeypatch, G, heights, lambda: G.migrate(s, G.RunOptions(), list(range(1, shots + 1)), v, rho)))


# 8-row tiles either side of the length up to which a launch takes one row per thread: 294 and 300
# tiles in a merged launch, 147 and 150 in one kernel's
@pytest.mark.gpu
@pytest.mark.parametrize("Z", [392, 400])
@pytest.mark.parametrize("accum", [0, 1, 2])
@pytest.mark.parametrize("heights", [(8, 8, 8, 8), (16, 8, 8, 16)])
def test_pipelined_form_of_eight_rows_either_side_of_two_tiles_per_sm(rtmlib, monkeypatch, Z, accum, heights):
    G = rtmlib
    nx, nz, npml = 344, Z - 40, 20
    v, rho = _models(nz, nx, Z)
    s = _survey(G, nx, nz, npml, 60, receiver_depth=2)
    _same(*_both(monkeypatch, G, heights, lambda: G.migrate(s, G.RunOptions(accum_fp64=accum), [1], v, rho)))


# 12-row tiles, which the one-column kernels do not have: with every tile on the general body all
# heights round alike; the interior body of the forward pressure fuses one product (compared with the
# tolerance of test_gpu_parity, 1e-4).  Depths that leave 1, 8 and 11 rows in the last tile, padded
# lengths at the end of the damping factors' padding (64 rows), both strip types and accumulators
@pytest.mark.gpu
@pytest.mark.parametrize("X,Z,npml,accum", [(384, 133, 20, 0), (513, 128, 21, 1), (400, 191, 10, 2), (60, 64, 12, 0),
                                            (390, 320, 33, 3)])
@pytest.mark.parametrize("heights", [(12, 12, 12, 12), (16, 16, 12, 8)])
def test_pipelined_form_at_twelve_rows(rtmlib, monkeypatch, X, Z, npml, accum, heights):
    G = rtmlib
    nx, nz = X - 2 * npml, Z - 2 * npml
    v, rho = _models(nz, nx, X + Z)
    s = _survey(G, nx, nz, npml, 90)
    o = G.RunOptions(accum_fp64=accum, strip_precision="fp16" if accum == 2 else "fp32")
    run = lambda: G.migrate(s, o, [1, 3], v, rho)
    monkeypatch.setenv("RTM_B200_FAST_TILES", "0")
    monkeypatch.setenv("RTM_B200_KERNELS", "scalar")
    for k in ("VEL", "VEL_RECON", "PRES", "PRES_RECON"):
        monkeypatch.setenv("RTM_B200_BZ_" + k, "16")
    want = run()
    monkeypatch.setenv("RTM_B200_KERNELS", "vector")
    for k, h in zip(("VEL", "VEL_RECON", "PRES", "PRES_RECON"), heights):
        monkeypatch.setenv("RTM_B200_BZ_" + k, str(h))
    _same(want, run())
    monkeypatch.delenv("RTM_B200_FAST_TILES")
    got = run()
    for k in ("image1", "image2s", "illum"):
        a, b = got[k].astype(np.float64), want[k].astype(np.float64)
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), k


@pytest.mark.gpu
def test_twelve_rows_need_the_pipelined_form(rtmlib, monkeypatch):
    v, rho = _models(60, 60, 0)
    monkeypatch.setenv("RTM_B200_KERNELS", "scalar")
    monkeypatch.setenv("RTM_B200_BZ_PRES", "12")
    with pytest.raises(rtmlib.RtmError):
        rtmlib.migrate(_survey(rtmlib, 60, 60, 12, 30), rtmlib.RunOptions(), [1], v, rho)


# chunk boundaries of the host copies: images of one chunk (2^18 floats), one cell less and more,
# a small one and several chunks; fp64 images narrowed on the way; fields with row pitch
@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz", [(4096, 64), (4095, 64), (4097, 64), (50, 30), (2300, 400)])
@pytest.mark.parametrize("accum", [0, 1])
def test_images_and_fields_to_the_host(rtmlib, nx, nz, accum):
    cudart = C.CDLL("libcudart.so.12")
    cudart.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    G = rtmlib
    v, rho = _models(nz, nx, nx)
    s = _survey(G, nx, nz, 10, 30)
    with G.Session(s, G.RunOptions(accum_fp64=accum), [1], v, rho) as ss:
        ss.run()
        got, ptrs = ss.images(), ss.image_ptrs()
        for k, p in ptrs.items():   # the device array through the driver's own copy
            want = np.empty(nx * nz, np.float64 if accum else np.float32)
            assert cudart.cudaMemcpy(want.ctypes.data, p, want.nbytes, 2) == 0
            assert np.array_equal(got[k].ravel(), want.astype(np.float32)), k
        if accum:
            f = ss.images_f64()
            for k in f:
                assert np.array_equal(got[k], f[k].astype(np.float32)), k
        ps, _ = ss.wavefields(0, nx + 20, nz + 20)
    p = G.forward(s, G.RunOptions(), 1, v, rho, 30)[0]
    assert p.shape == (nz + 20, nx + 20) and np.isfinite(ps).all() and np.abs(p).max() > 0
    with G.Session(s, G.RunOptions(), [1], v, rho) as ss:   # the same field through another copy
        ss.model()
        assert np.array_equal(ss.wavefields(0, nx + 20, nz + 20)[0], p)


# the other imaging conditions take words of four columns: interiors that start and end at every
# alignment, one word and partial last words, against the oracle
@pytest.mark.gpu
@pytest.mark.parametrize("nx,npml", [(61, 20), (62, 21), (63, 22), (64, 23), (125, 12), (129, 13), (3, 10)])
@pytest.mark.parametrize("accum", [0, 1])
def test_other_imaging_conditions_at_word_edges(rtmlib, oracle, nx, npml, accum):
    G = rtmlib
    nz = 41
    v, rho = _models(nz, nx, nx)
    s = _survey(G, nx, nz, npml, 130, spx0=(nx // 2) * 10.0, amp=1.0e4)
    got = G.migrate(s, G.RunOptions(extra_images=1, accum_fp64=accum), [1], v, rho)
    d = {k: getattr(s, k) for k in s.__dataclass_fields__}
    want = oracle.rtm_model(d, [1], v, rho, extra=1)
    # the tolerances of test_gpu_parity: 1e-4 where the terms are sums of products, 3e-3 where they
    # switch on signs of rounded products
    for k, tol in (("image1", 1e-4), ("image5s", 1e-4), ("image5m", 1e-4), ("image3m", 3e-3)):
        a, b = got[k].astype(np.float64), want[k].astype(np.float64)
        assert np.linalg.norm(b) > 0 and np.linalg.norm(a - b) <= tol * np.linalg.norm(b), k
