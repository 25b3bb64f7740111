"""The device memory that MTF and NNPS calls keep between them: shared by
threads, grown, given back, and forgotten with its context."""
import os
import subprocess
import sys
import textwrap
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from hybridmantis_b200 import analysis
from oracle import analysis_oracle as ao

pytestmark = pytest.mark.gpu


def _mtf(shape):
    img = np.random.default_rng(shape[0]).gamma(2.0, 3.0, shape)
    want = ao.mtf(img, 1.0, 20)

    def call():
        got = analysis.mtf(img, 1.0, 20)
        return all(np.allclose(got[k], w, rtol=1e-9, atol=1e-12)
                   for k, w in zip(("freq", "mtf_x", "mtf_y", "mtf_r"), want))
    return call


def _nnps(n, side, roi):
    imgs = np.random.default_rng(side).poisson(200.0, (n, side, side)).astype(np.float64)
    _, nr, n2, _ = ao.nnps(imgs, 1.0, roi, 0, 0, 2, 2, 9)

    def call():
        got = analysis.nnps(imgs, 1.0, roi, 0, 0, 2, 2, 9)
        return np.allclose(got["nnps_r"], nr, rtol=1e-9) and np.allclose(got["nnps_2d"], n2, rtol=1e-9, atol=1e-12 * n2.max())
    return call


def test_threads_with_calls_of_every_size(require_gpu):
    """Every call of every thread gives the oracle's result: calls that share the
    kept memory, that grow it, that run beside another, and one too large for it
    (4 images of 1,500 x 1,500: 144 MiB).  An exception in a thread fails here."""
    analysis.release()
    calls = [_mtf((90, 70)), _mtf((331, 512)), _nnps(2, 70, 32), _nnps(4, 1500, 750)]
    times = [40, 20, 40, 3]

    def work(call, n):
        return [call() for _ in range(n)]

    with ThreadPoolExecutor(len(calls)) as ex:
        jobs = [ex.submit(work, c, n) for c, n in zip(calls, times)]
        done = [j.result() for j in jobs]
    assert [len(d) for d in done] == times
    assert all(all(d) for d in done)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_release_gives_the_memory_back(require_gpu):
    small, large = _mtf((90, 70)), _nnps(4, 1024, 512)  # 32 MiB of images and 32 MiB of transforms
    assert small() and large()
    kept = _free()
    analysis.release()
    assert _free() >= kept + (60 << 20)
    analysis.release()  # nothing to give back
    assert small() and large()


def test_release_beside_calls(require_gpu):
    call = _mtf((90, 70))
    with ThreadPoolExecutor(2) as ex:
        job = ex.submit(lambda: [call() for _ in range(60)])
        while not job.done():
            analysis.release()
        assert all(job.result())


def test_a_context_reset_between_calls(require_gpu):
    """The caller may reset the device's context: no handle of the old one is
    used, and the next call works again or reports an error."""
    code = textwrap.dedent("""
        import ctypes, numpy as np
        from hybridmantis_b200 import analysis
        img = np.random.default_rng(1).gamma(2.0, 3.0, (90, 70))
        want = analysis.mtf(img, 1.0, 20)["mtf_r"]
        cuda = ctypes.CDLL("libcuda.so.1")
        dev = ctypes.c_int()
        assert cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert cuda.cuDevicePrimaryCtxReset_v2(dev) == 0
        for _ in range(2):
            try:
                assert np.array_equal(analysis.mtf(img, 1.0, 20)["mtf_r"], want)
                print("result")
            except RuntimeError as e:
                print("error:", e)
        print("end")
    """)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stdout.rstrip().endswith("end"), r.stdout + r.stderr
    print(r.stdout)
