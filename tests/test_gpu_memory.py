"""Device memory kept between calls (csrc/device_memory.h) on the GPU: reuse by calls
of other sizes, a failed call, and giving it back."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(capi, pkg):
    """Calls of different sizes and kinds, and what each returns."""
    out = []
    for side, nt, bs, kw in ((48, 17, 4, {}), (21, 9, 3, dict(traj_length=7)), (64, 16, 8, {}),
                             (32, 16, 4, dict(optimize_pgure=0, lambda_=0.1)), (96, 16, 4, {})):
        noisy, _, (a, m, s) = pkg.synth.workload("arps_256", seed=side, side=side, nt=nt)
        p = capi.default_params(block_size=bs, median_size=-1, random_seed=3, alpha=a / 300,
                                mu=m / 300, sigma=s / 300, **kw)
        Y, est, _, ex = capi.denoise_ex(noisy, p, features=True)
        out += [Y, est, ex["risk"], ex["features"]]
    rng = np.random.default_rng(2)
    out.append(capi.hot_pixel_filter(rng.integers(0, 65536, (50, 70, 3), dtype=np.uint16), 2.0))
    f = rng.normal(size=(700, 67)).astype(np.float32)
    m = pkg.learned.init_model(f, rng.uniform(-6, 0, 700).astype(np.float32), seed=1)
    out.append(capi.lambda_predict(m, f))
    return out


def test_results_do_not_depend_on_what_ran_before(capi, pkg):
    capi.release_memory()
    first = _calls(capi, pkg)
    for _ in range(2):  # on blocks with other calls' contents
        for x, y in zip(_calls(capi, pkg), first):
            np.testing.assert_array_equal(x, y)


def test_calls_after_a_failed_one(capi, pkg):
    """One impossible allocation (575 GB) ends a call in the middle of its arrays."""
    first = _calls(capi, pkg)
    one = np.zeros(capi.LAMBDA_MODEL_FLOATS, np.float32)
    ptr = ctypes.c_void_p(one.ctypes.data)  # not read: the allocation comes first
    assert capi.load().pgsvt_lambda_predict(ptr, ptr, 2 ** 31, ptr) == capi.ERR_OOM
    for x, y in zip(_calls(capi, pkg), first):
        np.testing.assert_array_equal(x, y)


def test_memory_is_given_back(capi, pkg):
    """All of it, also when another thread asks."""
    import torch
    first = _calls(capi, pkg)
    capi.release_memory()
    free0 = torch.cuda.mem_get_info()[0]
    _calls(capi, pkg)
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept > 0
    t = threading.Thread(target=capi.release_memory)
    t.start()
    t.join()
    assert torch.cuda.mem_get_info()[0] >= free0
    for x, y in zip(_calls(capi, pkg), first):
        np.testing.assert_array_equal(x, y)


def test_concurrent_calls_and_releases(capi, pkg):
    """Calls of different sizes on four threads, blocks changing hands between them,
    while a fifth keeps giving the memory back: every result is that of a call alone."""
    first = _calls(capi, pkg)
    wrong, stop = [], threading.Event()

    def work():
        try:
            for _ in range(3):
                for k, (x, y) in enumerate(zip(_calls(capi, pkg), first)):
                    if not np.array_equal(x, y):
                        wrong.append(k)
        except Exception as e:  # reported by the main thread
            wrong.append(e)

    def give_back():
        while not stop.wait(0.002):
            capi.release_memory()

    threads = [threading.Thread(target=work) for _ in range(4)]
    giver = threading.Thread(target=give_back)
    for t in threads + [giver]:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    giver.join()
    assert not wrong
