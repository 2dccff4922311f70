"""Launch plans only reorganise the work: on grids with interior tiles (128 columns that hold no
PML, source or receiver cell) the tile heights, the interior body, the kernel form, the batching, the
tuner and a resumed run give the same bits."""
import numpy as np
import pytest

NX, NZ, NPML, SHOTS = 420, 130, 20, [1, 2, 3]
IMAGES = ("image1", "image2s", "illum")
EXTRA = ("image3s", "image4s", "image5s", "imagetrue")


def _models(nz, nx, seed):
    rng = np.random.default_rng(seed)
    v = 1800 + 6 * np.arange(nz)[:, None] + 150 * rng.random((nz, nx))
    return np.minimum(v, 3800).astype(np.float32), (2000 + 100 * rng.random((nz, nx))).astype(np.float32)


def _survey(G, nx=NX, nz=NZ, npml=NPML, nt=300, **kw):
    d = dict(nx=nx, nz=nz, nt=nt, dx=10.0, dz=10.0, dt=float(np.float32(1e-3)), npml=npml, fdom=25.0, layout=2,
             spx0=(nx // 3) * 10.0, spz0=20.0, dspx=10.0, mode=0, mute=0)
    d.update(kw)
    return G.SurveyConfig(**d)


def _heights(*h):
    return {"RTM_B200_BZ_" + k: str(x) for k, x in zip(("VEL", "VEL_RECON", "PRES", "PRES_RECON"), h)}


def _run(G, monkeypatch, env, options):
    with monkeypatch.context() as m:
        for k in ("RTM_B200_TUNE", "RTM_B200_TUNE_CACHE", "RTM_B200_KERNELS", *_heights(0, 0, 0, 0)):
            m.delenv(k, raising=False)
        for k, x in env.items():
            m.setenv(k, x)
        return G.migrate(_survey(G), G.RunOptions(**options), SHOTS, *_models(NZ, NX, 3))


def _same(a, b, keys=IMAGES):
    for k in keys:
        assert np.abs(b[k]).max() > 0 and np.array_equal(a[k], b[k]), k
    for x, y in zip(a["gathers"], b["gathers"]):
        assert np.array_equal(x, y)


PLANS = {
    "8 merged": _heights(8, 8, 8, 8), "16 merged": _heights(16, 16, 16, 16), "12 merged": _heights(12, 12, 12, 12),
    "16/16/12/8": _heights(16, 16, 12, 8), "16/16/8/8": _heights(16, 16, 8, 8), "32": _heights(32, 32, 32, 32),
    "64/16/64/16": _heights(64, 16, 64, 16), "general body": dict(_heights(8, 8, 8, 8), RTM_B200_FAST_TILES="0"),
    "one column, 8": dict(_heights(8, 8, 8, 8), RTM_B200_KERNELS="scalar"),
    "one column, 32/16/16": dict(_heights(32, 16, 16, 16), RTM_B200_KERNELS="scalar"),
    "one column, general body": dict(_heights(32, 16, 16, 16), RTM_B200_KERNELS="scalar", RTM_B200_FAST_TILES="0"),
    "tuner": {}, "no tuner": {"RTM_B200_TUNE": "0"},
}


@pytest.mark.gpu
def test_plans_give_one_set_of_bits_on_wide_grids(rtmlib, monkeypatch):
    want = _run(rtmlib, monkeypatch, PLANS["one column, general body"], {})
    others = {"whole step": {"RTM_B200_FUSED": "1", "RTM_B200_TZ_STEP": "16"}, "persistent": {"RTM_B200_PERSIST": "1"}}
    for name, env in {**PLANS, **others}.items():
        try:
            _same(_run(rtmlib, monkeypatch, env, {}), want)
        except AssertionError as e:
            raise AssertionError(name) from e


# with the other imaging conditions the pressure height is part of the result, and follows from the
# session's shots alone
@pytest.mark.gpu
@pytest.mark.parametrize("accum,extra", [(0, 0), (1, 0), (0, 1)])
def test_batching_and_resume_give_one_set_of_bits_on_wide_grids(rtmlib, monkeypatch, tmp_path, accum, extra):
    G = rtmlib
    options = dict(accum_fp64=accum, extra_images=extra)
    keys = IMAGES + EXTRA if extra else IMAGES
    want = _run(G, monkeypatch, PLANS["no tuner"], options)
    for batch in (0, 1, 2):
        _same(_run(G, monkeypatch, {}, dict(options, batch=batch)), want, keys)
    for env in ({"RTM_B200_TUNE": "0", "RTM_B200_KERNELS": "scalar"}, {"RTM_B200_PERSIST": "1"}):
        _same(_run(G, monkeypatch, env, options), want, keys)
    v, rho = _models(NZ, NX, 3)
    path = str(tmp_path / "run.ckpt")
    with G.Session(_survey(G), G.RunOptions(batch=2, **options), SHOTS, v, rho) as a:
        a.run_range(0, 2)
        a.save_checkpoint(path, 2)
    monkeypatch.setenv("RTM_B200_TUNE", "0")   # the rest under another plan
    with G.Session(_survey(G), G.RunOptions(batch=2, **options), SHOTS, v, rho) as b:
        assert b.load_checkpoint(path) == 2
        b.run_range(2, 1)
        got = {**b.images(), **(b.images_extra() if extra else {})}
    for k in keys:
        assert np.array_equal(got[k], want[k]), k


# shots that fill more than 6 million cells together and fewer one by one: the line where that height
# changes
@pytest.mark.gpu
def test_the_other_conditions_height_does_not_follow_the_batch(rtmlib):
    G = rtmlib
    nx, nz, shots = 1400, 1000, [1, 2, 3, 4, 5]
    v, rho = _models(nz, nx, 5)
    out = []
    for batch in (0, 2, 1):
        with G.Session(_survey(G, nx=nx, nz=nz, nt=40), G.RunOptions(batch=batch, extra_images=1), shots, v, rho) as ss:
            ss.run()
            out.append(({**ss.images(), **ss.images_extra()}, [ss.gather(k) for k in range(5)], ss.tile_heights()["pres"]))
    assert [o[2] for o in out] == [16, 16, 16]
    for images, gathers, _ in out[1:]:
        for k in IMAGES + EXTRA:
            assert np.abs(images[k]).max() > 0 and np.array_equal(images[k], out[0][0][k]), k
        for a, b in zip(gathers, out[0][1]):
            assert np.array_equal(a, b)


@pytest.mark.gpu
def test_modelling_before_and_after_the_tuner_gives_the_same_gathers(rtmlib):
    G = rtmlib
    with G.Session(_survey(G), G.RunOptions(), SHOTS, *_models(NZ, NX, 3)) as ss:
        ss.model()
        before = [ss.gather(k) for k in range(len(SHOTS))]
        ss.run()
        ss.model()
        for k, g in enumerate(before):
            assert np.abs(g).max() > 0 and np.array_equal(ss.gather(k), g)


# a batch of more than 400 MB of fields, whose tiles keep the order of the fields (smaller ones start with
# the tiles that take longest), in merged and in separate launches
@pytest.mark.gpu
@pytest.mark.parametrize("heights", [(8, 8, 8, 8), (16, 16, 8, 8), (16, 16, 12, 8)])
def test_large_batches_in_field_order(rtmlib, monkeypatch, heights):
    G = rtmlib
    nx, nz, shots = 350, 960, list(range(1, 27))   # 26 shots of 10 arrays of 416 x 1000 floats
    v, rho = _models(nz, nx, 26)
    out = []
    for env in ({"RTM_B200_KERNELS": "scalar", "RTM_B200_TUNE": "0"}, _heights(*heights)):
        with monkeypatch.context() as m:
            for k, x in env.items():
                m.setenv(k, x)
            out.append(G.migrate(_survey(G, nx=nx, nz=nz, nt=40), G.RunOptions(), shots, v, rho))
    _same(out[1], out[0])
