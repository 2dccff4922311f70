"""Read-back of images, gathers and fields (rtm_copy.cu): its order behind a caller's own work on the
device arrays."""
import numpy as np
import pytest


def _models(nz, nx, seed):
    rng = np.random.default_rng(seed)
    v = 1800 + 6 * np.arange(nz)[:, None] + 150 * rng.random((nz, nx))
    return np.minimum(v, 3800).astype(np.float32), (2000 + 100 * rng.random((nz, nx))).astype(np.float32)


def _survey(G, nx, nz, npml, nt, **kw):
    d = dict(nx=nx, nz=nz, nt=nt, dx=10.0, dz=10.0, dt=float(np.float32(1e-3)), npml=npml, fdom=25.0, layout=2,
             spx0=(nx // 3) * 10.0, spz0=20.0, dspx=10.0, mode=0, mute=0)
    d.update(kw)
    return G.SurveyConfig(**d)


class _DeviceArray:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


# images of several chunks (fp32, and fp64 narrowed on the way) and of less than a quarter of one
@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz", [(600, 300), (160, 60)])
@pytest.mark.parametrize("accum,f64", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("blocking_stream", [False, True])
def test_images_wait_for_work_on_the_default_stream(rtmlib, nx, nz, accum, f64, blocking_stream):
    import torch

    G = rtmlib
    v, rho = _models(nz, nx, nx)
    with G.Session(_survey(G, nx, nz, 12, 30), G.RunOptions(accum_fp64=accum), [1], v, rho) as ss:
        ss.run()
        t = torch.as_tensor(_DeviceArray(ss.image_ptrs()["image1"], nx * nz, "<f8" if accum else "<f4"), device="cuda")
        want = t.cpu().numpy() + 1
        torch.cuda.synchronize()
        # queued behind a pause of some 50 ms: in the default stream, or in one that synchronises with it
        if blocking_stream:
            import ctypes as C
            rt, h = C.CDLL("libcudart.so.12"), C.c_void_p()
            assert rt.cudaStreamCreate(C.byref(h)) == 0
            st = torch.cuda.ExternalStream(h.value)
        else:
            st = torch.cuda.default_stream()
        with torch.cuda.stream(st):
            torch.cuda._sleep(100_000_000)
            t.add_(1)
        got = (ss.images_f64() if f64 else ss.images())["image1"].ravel()
        torch.cuda.synchronize()
        assert np.array_equal(got, want if f64 else want.astype(np.float32))


RESET = """
import ctypes as C
import numpy as np
import gubingluo_b200 as G

def context():
    f, q, n = C.c_void_p(), C.c_int(), C.c_ulonglong()
    assert rt.cudaGetDriverEntryPoint(b"cuCtxGetId", C.byref(f), C.c_ulonglong(0), C.byref(q)) == 0
    assert C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)(f.value)(None, C.addressof(n)) == 0
    return n.value

G.lib()
rt = C.CDLL("libcudart.so.12")
obs = np.random.default_rng(0).standard_normal((400, 200)).astype(np.float32)
a = G.interp_gather(obs, 399, 400, 1e-3, 1e-3)   # 638 KB: through the kept buffers
before = context()
assert rt.cudaDeviceReset() == 0
assert rt.cudaSetDevice(0) == 0 and rt.cudaFree(None) == 0
assert context() != before, "a new context must have a new number: stopping before the next copy"
assert np.array_equal(G.interp_gather(obs, 399, 400, 1e-3, 1e-3), a)
print("same")
"""


@pytest.mark.gpu
def test_results_after_a_device_reset(rtmlib):
    """In a process of its own: cudaDeviceReset ends the process's context."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
