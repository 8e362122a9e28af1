"""Staged model uploads: the ring of slots on the CPU (a worker stands for the device's copy
engine), and whole runs on a stream whose handle means another stream on other threads."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "fomo.jl_b200" / "csrc"

HARNESS = r"""
#include <atomic>
#include <chrono>
#include <cstring>
#include <deque>
#include "staging.h"
// The "device" copies a slot some time after its copy was issued; a slot refilled
// before that shows in dst.
extern "C" int run(int n, int slots, int helpers, int chunk, int fail_at, const char* src, char* dst,
                   int* foreign, int* disorder) {
  std::vector<char> ring((size_t)slots * chunk);
  std::mutex mu;
  std::condition_variable cv;
  std::deque<int> queue;
  std::vector<int> pending(slots, 0);
  bool stop = false;
  std::thread device([&] {
    std::unique_lock<std::mutex> lk(mu);
    for (;;) {
      cv.wait(lk, [&] { return stop || !queue.empty(); });
      if (queue.empty()) return;
      const int k = queue.front();
      queue.pop_front();
      lk.unlock();
      std::this_thread::sleep_for(std::chrono::microseconds(100 * (k % 5)));
      std::memcpy(dst + (size_t)k * chunk, ring.data() + (size_t)(k % slots) * chunk, chunk);
      lk.lock();
      --pending[k % slots];
      cv.notify_all();
    }
  });
  const auto me = std::this_thread::get_id();
  int last = -1;
  *foreign = *disorder = 0;
  const int rc = fomo::staged_copy(
      n, slots, helpers,
      [&](size_t s) {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return pending[s] == 0; });
        return 0;
      },
      [&](size_t k, size_t s) {
        if ((int)k == fail_at) return 7;
        std::memcpy(ring.data() + s * chunk, src + k * chunk, chunk);
        return 0;
      },
      [&](size_t k, size_t s) {
        *foreign += std::this_thread::get_id() != me;
        *disorder += (int)k != last + 1 || s != k % slots;
        last = (int)k;
        std::lock_guard<std::mutex> lk(mu);
        ++pending[s];
        queue.push_back((int)k);
        cv.notify_all();
        return (int)k == -fail_at ? 9 : 0;
      });
  {
    std::lock_guard<std::mutex> lk(mu);
    stop = true;
    cv.notify_all();
  }
  device.join();
  return rc;
}
"""


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("staging")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-shared", "-fPIC", "-I", str(CSRC), "-o",
                    str(d / "h.so"), str(d / "h.cpp")], check=True)
    lib = C.CDLL(str(d / "h.so"))

    def run(n, slots, helpers, fail_at=10 ** 6, chunk=512):
        src = np.random.default_rng(n).integers(0, 255, max(n, 1) * chunk).astype(np.uint8)
        dst = np.zeros_like(src)
        foreign, disorder = C.c_int(-1), C.c_int(-1)
        rc = lib.run(n, slots, helpers, chunk, fail_at, src.ctypes.data_as(C.c_void_p),
                     dst.ctypes.data_as(C.c_void_p), C.byref(foreign), C.byref(disorder))
        return rc, np.array_equal(src[:n * chunk], dst[:n * chunk]), foreign.value, disorder.value

    return run


@pytest.mark.parametrize("helpers", [0, 1, 4, 9])
@pytest.mark.parametrize("n,slots", [(0, 8), (1, 8), (7, 8), (8, 8), (9, 8), (83, 8), (40, 1)])
def test_slots_carry_every_chunk_and_only_the_caller_issues(ring, n, slots, helpers):
    assert ring(n, slots, helpers) == (0, True, 0, 0)


@pytest.mark.parametrize("helpers", [0, 1, 4])
def test_first_error_ends_the_copy(ring, helpers):
    rc, same, foreign, _ = ring(50, 8, helpers, fail_at=21)
    assert (rc, same, foreign) == (7, False, 0)
    rc, same, foreign, _ = ring(50, 8, helpers, fail_at=-21)
    assert (rc, same, foreign) == (9, False, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("handle", [1, 2])  # cudaStreamLegacy, cudaStreamPerThread
def test_staged_upload_on_a_callers_stream(fomo, handle):
    """Pageable models over 16 MB: what reads them must run after the copies."""
    from fomo_b200 import _lib as L

    nx, nz = 3001, 2003
    rng = np.random.default_rng(7)
    vp = rng.uniform(2000, 3000, (nx, nz)).astype(np.float32, order="F")
    rho = rng.uniform(1500, 2500, (nx, nz)).astype(np.float32, order="F")
    rx = np.linspace(1, nx, 300).astype(int)
    kw = dict(sx=rx, sz=np.full(300, nz - 1), rx=rx, rz=np.full(300, nz), nbc=4, fd_order=2)
    ref = fomo.acoustic2d(vp, rho, 10.0, 1e-3, 4, 15.0, **kw)
    ctx = L.context(0)
    ctx.set_stream(handle)
    try:
        for _ in range(5):
            vp2 = np.asfortranarray(vp[::-1] + np.float32(1.0))  # other models in the same workspace
            fomo.acoustic2d(vp2, rho, 10.0, 1e-3, 4, 15.0, **kw)
            a = fomo.acoustic2d(vp, rho, 10.0, 1e-3, 4, 15.0, **kw)
            assert np.array_equal(a.seis_p, ref.seis_p)
            assert np.array_equal(a.seis_vz, ref.seis_vz)
    finally:
        ctx.set_stream(None)
    assert np.abs(ref.seis_p).max() > 0
